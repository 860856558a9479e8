"""The 2-CTA register-FFT slice kernel at the sizes and thread counts it is
launched with: 64 x 64, and 128 x 96 with at most one CTA per SM (384 threads) and
with more (256), flux rows included.  Against the CPU oracle after a few steps:
complex64 rounding is about 1e-7 a step, so psi agrees to 1e-4 with room and P(E)
to the complex64 contract of 1e-3.
"""
import numpy as np
import pytest

from oracle import pyoracle as O
from qd_b200 import systems as S, QD_PREC_FP32, QD_PREC_FP64
from qd_b200.timeevolution import Propagator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,nth,runs", [(64, 64, 12, 1), (128, 96, 10, 1), (128, 96, 25, 3),
                                            (128, 96, 24, 4)])
def test_pair_of_ctas(n1, n2, nth, runs, monkeypatch):
    monkeypatch.setenv("QD_SLICE_CLUSTER", "9")
    base = S.build_case("f+h2", n1, n2, nth, m=nth - 1, total_steps=4, n_energies=5,
                        n_gradient_points=5, precision=QD_PREC_FP32)
    data = [S.copy_case(base) for _ in range(runs)]
    for r, d in enumerate(data):
        d.psi *= 1.0 + 0.25 * r
    want = []
    for d in data:
        a = S.copy_case(d)
        a.options.precision = QD_PREC_FP64
        _, e = O.oracle_time_evolution(a, energies=True)
        want.append((a, e))
    with Propagator(data) as p:
        p.set_energy_interval(2)
        p.propagate(4)
        logs = [p.energy_log(r) for r in range(runs)]
        p.download()
    for d, (a, e), log in zip(data, want, logs):
        assert np.abs(d.psi - a.psi).max() < 1e-4 * np.abs(a.psi).max()
        assert np.abs(d.CRP.CRP - a.CRP.CRP).max() < 1e-3
        for row in log:
            ref = e[int(row[0]) - 1]
            assert np.abs(row[1:] - ref).max() <= 1e-4 * np.abs(ref).max()
