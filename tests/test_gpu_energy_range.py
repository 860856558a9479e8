"""The energies of a step on the run-time complex64 l-space kernels square the
wavepacket's values in FP64: a wavepacket scaled by 2^-66, whose squares complex64
cannot hold (2^-132), has 2^-132 of the energies.  Scaling by a power of two
commutes with every rounding except of values below 2^-126, 2^-60 of the largest
ones here, and the sums are FP64 in an order of their own: 1e-12 relative.
"""
import numpy as np
import pytest

from qd_b200 import systems as S, QD_PREC_FP32
from qd_b200.timeevolution import Propagator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2", [(18, 20), (36, 48), (54, 200)])
def test_energies_of_a_small_wavepacket(n1, n2, monkeypatch):
    monkeypatch.setenv("QD_SLICE_CLUSTER", "12")
    monkeypatch.setenv("QD_COLUMN_PATH", "simt")
    logs = []
    for scale in (1.0, 2.0 ** -66):
        d = S.build_case("h+h2", n1, n2, 8, m=7, total_steps=4, n_energies=5, n_gradient_points=3)
        d.options.precision = QD_PREC_FP32
        d.psi *= scale
        with Propagator(d) as p:
            p.set_energy_interval(2)
            p.propagate(4)
            logs.append(p.energy_log()[:, 1:4] / scale / scale)
    assert logs[0].shape == (2, 3) and np.all(logs[0][:, 0] > 0)
    assert np.abs(logs[1] - logs[0]).max() < 1e-12 * np.abs(logs[0]).max()
