"""The run-time register-FFT l-space kernels (a row and a column launch) against
the CPU oracle: every radix and group of radices in both directions, sizes that do not fill a block of rows or of columns, the largest sizes they take, batches of
several bases, and the energies of the step.  FP64 to 1e-10 relative (its
contract; a step's rounding is of order 1e-15), complex64 to 1e-4 after a few
steps (its kernels differ from FP64 by about 1e-7 a step).
"""
import numpy as np
import pytest

from oracle import pyoracle as O
from qd_b200 import systems as S, QD_PREC_FP32, QD_PREC_FP64
from qd_b200.timeevolution import Propagator

pytestmark = pytest.mark.gpu

# FP64: 4 x 4, 5 x 4, 6 x 5, 8 x 6, 9 x 8, 10 x 9, 12 x 10, 15 x 12, 16 x 15, 16 x 16, 18 x 12, 20 x 10;
# complex64: single radices and the pairs 2 3, 2 5, 3 3, 3 5, 4 3, 4 5, 5 5, 8 2, 8 3, 8 4
GRIDS = [(16, 20), (30, 48), (72, 90), (120, 54), (54, 120), (180, 16), (16, 240), (256, 24),
         (24, 256), (216, 40), (40, 200), (108, 100), (150, 36), (250, 10), (10, 250)]


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def check(runs, steps, every, monkeypatch, prec, tol):
    monkeypatch.setenv("QD_SLICE_CLUSTER", "12")
    want, energies = [], []
    for d in runs:
        a = S.copy_case(d)
        a.options.precision = QD_PREC_FP64
        _, e = O.oracle_time_evolution(a, energies=True)
        want.append(a)
        energies.append(e)
    for d in runs:
        d.options.precision = prec
    with Propagator(runs) as p:
        p.set_energy_interval(every)
        p.propagate(steps)
        logs = [p.energy_log(r) for r in range(len(runs))]
        p.download()
    for d, a, e, log in zip(runs, want, energies, logs):
        assert rel(d.psi, a.psi) < tol
        assert np.abs(d.CRP.CRP - a.CRP.CRP).max() < (1e-8 if prec == QD_PREC_FP64 else 1e-3)
        for row in log:
            ref = e[int(row[0]) - 1][:3]
            assert np.abs(row[1:4] - ref).max() < tol * max(np.abs(ref).max(), 1e-3)


@pytest.mark.parametrize("prec,tol", [(QD_PREC_FP64, 1e-10), (QD_PREC_FP32, 1e-4)])
@pytest.mark.parametrize("n1,n2", GRIDS)
def test_grids(n1, n2, prec, tol, monkeypatch):
    d = S.build_case("h+h2", n1, n2, 6, m=5, total_steps=4, n_energies=5, n_gradient_points=3)
    check([d], 4, 2, monkeypatch, prec, tol)


@pytest.mark.parametrize("prec,tol", [(QD_PREC_FP64, 1e-10), (QD_PREC_FP32, 1e-4)])
def test_blocks_of_several_bases(prec, tol, monkeypatch):
    base = S.build_case("f+h2", 36, 30, 12, m=11, total_steps=6, n_energies=5, n_gradient_points=5)
    runs = [S.cs_case(base, J, K, 0, K + 1) for J, K in ((0, 0), (2, 1), (3, 3))]
    check(runs, 6, 3, monkeypatch, prec, tol)


def test_fp64_wide_column_tiles(monkeypatch):
    # enough slices for 16-column tiles, the last of them ragged (n1 = 72)
    d = S.build_case("h+h2", 72, 30, 64, m=59, total_steps=3, n_energies=5, n_gradient_points=3)
    check([d], 3, 3, monkeypatch, QD_PREC_FP64, 1e-10)
