"""Handles of different shapes stepped by several host threads at once, two and
two of them on the same kernel: every thread's wavepacket is bit for bit that of
a run by itself (psi involves no atomics).
"""
import threading

import numpy as np
import pytest

from qd_b200 import systems as S, QD_PREC_FP32, QD_PREC_FP64
from qd_b200.timeevolution import Propagator

pytestmark = pytest.mark.gpu

# column pass (72 and 128 angles), l-space columns and rows of either precision
SHAPES = [(QD_PREC_FP64, None, [(16, 20, 72), (16, 20, 128)]),
          (QD_PREC_FP64, None, [(16, 20, 8), (64, 240, 8)]),
          (QD_PREC_FP32, "12", [(18, 20, 8), (48, 250, 8)]),
          (QD_PREC_FP32, "1", [(16, 20, 8), (40, 60, 8)])]


def case(prec, n1, n2, nth):
    d = S.build_case("h+h2", n1, n2, nth, m=nth - 1, total_steps=400, n_energies=5,
                     n_gradient_points=3)
    d.options.precision = prec
    return d


def steps(p, calls):
    for _ in range(calls):
        p.propagate(100)


@pytest.mark.parametrize("prec,lines,shapes", SHAPES)
def test_shapes_in_threads(prec, lines, shapes, monkeypatch):
    if lines:
        monkeypatch.setenv("QD_SLICE_CLUSTER", lines)
    calls = 40
    alone = []
    for shape in shapes:
        d = case(prec, *shape)
        with Propagator(d) as p:
            steps(p, calls)
            p.download()
        alone.append(d.psi.copy())
    data = [case(prec, *s) for s in shapes]
    handles = [Propagator(d) for d in data]
    errors = []
    gate = threading.Barrier(len(handles))

    def work(p):
        gate.wait()
        try:
            steps(p, calls)
        except Exception as e:          # noqa: BLE001 -- reported by the test
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=(p,)) for p in handles]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for p, d, want in zip(handles, data, alone):
        p.download()
        p.close()
        np.testing.assert_array_equal(d.psi, want)
