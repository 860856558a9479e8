"""P(E) of the kernels whose launches prepare the flux rows (extra CTAs of the
run-time l-space row launches, extra clusters of the 2-CTA slice kernel), and of
the FP64 tensor-core column pass that writes those rows, on wavepackets that have
flux: random values everywhere, incoming amplitudes of 1, against the CPU oracle
relative to the largest |P(E)|.  FP64 1e-10 (its contract; a step's rounding is of
order 1e-15); complex64 1e-4 (about 1e-7 a step in psi, twice that in the
flux).  Each case first shows on the oracle that leaving out the last step's rows
would move P(E) by a hundred tolerances.
"""
import numpy as np
import pytest

from oracle import pyoracle as O
from qd_b200 import systems as S, QD_PREC_FP32, QD_PREC_FP64
from qd_b200.timeevolution import Propagator

pytestmark = pytest.mark.gpu

BOTH = [(QD_PREC_FP64, 1e-10), (QD_PREC_FP32, 1e-4)]


def dense(system, n1, n2, nth, points, seed, m=None):
    d = S.build_case(system, n1, n2, nth, m=nth - 1 if m is None else m, total_steps=4,
                     n_energies=7, n_gradient_points=points, r_surface=4.0)
    g = np.random.default_rng([seed, n1, n2, nth])
    d.psi = g.standard_normal(d.psi.shape) + 1j * g.standard_normal(d.psi.shape)
    d.CRP.eta_sq = np.ones(7)
    return d


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def check(runs, steps, prec, tol):
    want = []
    for d in runs:
        short, a = S.copy_case(d), S.copy_case(d)
        short.options.precision = a.options.precision = QD_PREC_FP64
        short.time.total_steps, a.time.total_steps = steps - 1, steps
        O.oracle_time_evolution(short)
        norms, energies = O.oracle_time_evolution(a, norms=True, energies=True)
        assert rel(short.CRP.CRP, a.CRP.CRP) > 100 * tol
        want.append((a, norms, energies))
        d.options.precision = prec
    with Propagator(runs if len(runs) > 1 else runs[0]) as p:
        p.set_energy_interval(2)
        p.propagate(steps - 1)
        p.propagate(1)
        got = [(p.norms(steps, r), p.energy_log(r)) for r in range(len(runs))]
        p.download()
    for d, (a, norms, energies), (n, log) in zip(runs, want, got):
        assert rel(d.psi, a.psi) < tol
        assert rel(d.CRP.CRP, a.CRP.CRP) < tol
        assert rel(n, norms) < tol
        for row in log:
            assert rel(row[1:4], energies[int(row[0]) - 1][:3]) < tol


# angles and columns that do and do not fill the flux CTAs
@pytest.mark.parametrize("prec,tol", BOTH)
@pytest.mark.parametrize("n1,n2,nth", [(16, 20, 6), (30, 48, 7), (72, 90, 5), (120, 54, 16), (250, 10, 3)])
def test_run_time_l_space(n1, n2, nth, prec, tol, monkeypatch):
    monkeypatch.setenv("QD_SLICE_CLUSTER", "12")
    check([dense("h+h2", n1, n2, nth, 5, 1)], 5, prec, tol)


@pytest.mark.parametrize("prec,tol", BOTH)
def test_run_time_l_space_batch(prec, tol, monkeypatch):
    monkeypatch.setenv("QD_SLICE_CLUSTER", "12")
    runs = []
    base = dense("f+h2", 36, 30, 12, 5, 2)
    for k, (J, K) in enumerate(((0, 0), (2, 1), (3, 3))):
        d = S.cs_case(base, J, K, 0, K + 1)
        d.psi = base.psi * (1.0 + 0.5j * k)
        d.CRP.eta_sq = np.ones(7)
        runs.append(d)
    check(runs, 6, prec, tol)


# the sizes past 256: FP64 up to 20 x 20, complex64 up to 32 x 25 points in two groups
@pytest.mark.parametrize("prec,tol,n1,n2", [
    (QD_PREC_FP64, 1e-10, 400, 16), (QD_PREC_FP64, 1e-10, 16, 400), (QD_PREC_FP64, 1e-10, 20, 320),
    (QD_PREC_FP64, 1e-10, 360, 300), (QD_PREC_FP32, 1e-4, 800, 10), (QD_PREC_FP32, 1e-4, 10, 800),
    (QD_PREC_FP32, 1e-4, 480, 12), (QD_PREC_FP32, 1e-4, 12, 600), (QD_PREC_FP32, 1e-4, 288, 360)])
def test_large_sizes(prec, tol, n1, n2, monkeypatch):
    monkeypatch.setenv("QD_SLICE_CLUSTER", "12")
    check([dense("h+h2", n1, n2, 4, 3, 3)], 3, prec, tol)


@pytest.mark.parametrize("n1,n2,nth,runs", [(64, 64, 12, 1), (128, 96, 10, 1), (128, 96, 25, 3)])
def test_pair_of_ctas(n1, n2, nth, runs, monkeypatch):
    monkeypatch.setenv("QD_SLICE_CLUSTER", "9")
    data = []
    base = dense("f+h2", n1, n2, nth, 5, 4)
    for r in range(runs):
        d = S.copy_case(base)
        d.psi = np.roll(base.psi, r, axis=2)
        data.append(d)
    check(data, 4, QD_PREC_FP32, 1e-4)


@pytest.mark.parametrize("nth,m", [(1, 0), (7, 6), (9, 5), (17, 16), (64, 63), (65, 64), (128, 127), (129, 128)])
def test_fp64_column_pass(nth, m):
    check([dense("h+h2", 18, 10, nth, 3, 5, m)], 5, QD_PREC_FP64, 1e-10)
