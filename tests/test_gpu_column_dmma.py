"""The FP64 column pass on the FP64 tensor cores at the edges of its tiles:
bases around multiples of eight (the mma groups) and sixteen (the shared-memory
rows), n_l above n_theta, grids whose columns do not fill a tile, the largest
basis it takes and the first one it leaves to the SIMT kernel, and batches whose
runs change basis from tile to tile.  Against the CPU oracle, 1e-10 relative
(the FP64 contract: a step adds rounding of order 1e-15).
"""
import numpy as np
import pytest

from oracle import pyoracle as O
from qd_b200 import systems as S
from qd_b200.timeevolution import Propagator

pytestmark = pytest.mark.gpu

EDGES = [(1, 0), (7, 6), (8, 8), (9, 5), (16, 15), (17, 16), (33, 28), (64, 63), (65, 64), (71, 40),
         (128, 127), (129, 128)]


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("nth,m", EDGES)
def test_basis_edges(nth, m):
    base = S.build_case("h+h2", 18, 10, nth, m=m, total_steps=8, n_energies=7, n_gradient_points=3)
    a, b = S.copy_case(base), S.copy_case(base)
    norms, _ = O.oracle_time_evolution(a, norms=True)
    with Propagator(b) as p:
        p.set_energy_interval(4)
        p.propagate(5)
        p.propagate(3)
        g, log = p.norms(8), p.energy_log()
        now = p.energies()
        p.download()
    assert rel(b.psi, a.psi) < 1e-10
    assert np.abs(g - norms).max() < 1e-10 * norms.max()
    assert np.abs(b.CRP.CRP - a.CRP.CRP).max() < 1e-8
    assert log[:, 0].tolist() == [4, 8] and np.all(np.isfinite(log)) and np.all(np.isfinite(now))


@pytest.mark.parametrize("nth", [24, 100])
def test_blocks_of_several_bases(nth):
    base = S.build_case("f+h2", 20, 12, nth, m=nth - 1, total_steps=6, n_energies=5,
                        n_gradient_points=5)
    runs = [S.cs_case(base, J, K, 0, K + 1) for J, K in ((0, 0), (2, 1), (2, 0), (3, 3), (2, 1))]
    want = []
    for d in runs:
        a = S.copy_case(d)
        O.oracle_time_evolution(a)
        want.append(a)
    with Propagator(runs) as p:
        p.propagate(6)
        p.download()
    for d, a in zip(runs, want):
        assert rel(d.psi, a.psi) < 1e-10
        assert np.abs(d.CRP.CRP - a.CRP.CRP).max() < 1e-8
