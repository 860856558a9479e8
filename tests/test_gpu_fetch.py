"""Results of the surface calls of every size and destination: small ones, ones
copied into pages that are in memory and ones staged into a fresh mapping (several
chunks, the last ragged) hold the same values, bit for bit, as the grid taken one
angle at a time.
"""
import ctypes as C
import mmap

import numpy as np
import pytest

from qd_b200 import _abi, systems as S
from qd_b200._abi import check, lib
from qd_b200.surrogate import Surrogate
from qd_b200.timeevolution import _grid_structs, leps_params

pytestmark = pytest.mark.gpu


def ptr(a):
    return a.ctypes.data_as(_abi.c_double_p)


def calls():
    fh = np.array([18.9984, 1.00783, 1.00783]) * S.AMU_ME
    hh = np.array([1.00783, 1.00783, 1.00783]) * S.AMU_ME
    p, sur = leps_params(S.leps_f_h2()), Surrogate(seed=3)
    return {
        "leps": lambda a, b, t, o: lib().qd_potential_leps(
            C.byref(a), C.byref(b), C.byref(t), ptr(fh), C.byref(p), 2.5, 0.4, 1, ptr(o)),
        "bkmp2": lambda a, b, t, o: lib().qd_potential_bkmp2(
            C.byref(a), C.byref(b), C.byref(t), ptr(hh), 2.5, 0.4, 1, ptr(o)),
        "mlp": lambda a, b, t, o: lib().qd_mlp_potential(
            sur._h, C.byref(a), C.byref(b), C.byref(t), ptr(fh), 2.5, 0.4, 1, ptr(o))}


@pytest.mark.parametrize("name", ["leps", "bkmp2", "mlp"])
@pytest.mark.parametrize("n1,n2,nth", [(90, 60, 8), (90, 60, 49), (131, 97, 83), (211, 161, 127)])
def test_destinations(name, n1, n2, nth):                # 0.3, 2.1, 8.4 and 34.5 MB
    R, r = np.linspace(0.5, 12.0, n1), np.linspace(0.4, 8.0, n2)
    x, _ = S.gauss_legendre(nth)
    f = calls()[name]
    want = np.zeros((nth, n2, n1))
    for k in range(nth):
        (a, b, t), keep = _grid_structs(R, r, x[k:k + 1])
        check(f(a, b, t, want[k]))
    (a, b, t), keep = _grid_structs(R, r, x)
    warm = np.full_like(want, np.nan)
    check(f(a, b, t, warm))
    pages = mmap.mmap(-1, want.nbytes, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    fresh = np.frombuffer(pages, dtype=np.float64).reshape(want.shape)
    check(f(a, b, t, fresh))
    np.testing.assert_array_equal(warm, want)
    np.testing.assert_array_equal(fresh, want)
