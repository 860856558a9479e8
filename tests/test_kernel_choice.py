"""qd_kernel_choice names the kernels that a handle runs, in either precision, and
the benchmark's line describes them from it."""
import ctypes as C
import os
import sys

import pytest

from conftest import REPO
from qd_b200 import systems as S, QD_PREC_FP32, QD_PREC_FP64

sys.path.insert(0, REPO)


@pytest.mark.gpu
@pytest.mark.parametrize("prec,n1,n2,nth,env,lines,column", [
    (QD_PREC_FP64, 64, 48, 16, None, 12, 1),
    (QD_PREC_FP64, 64, 48, 16, "0", 0, 1),          # the split kernels, asked for
    (QD_PREC_FP64, 12, 48, 16, None, 0, 1),         # a size with no two built radices
    (QD_PREC_FP64, 64, 48, 129, None, 12, 0),       # a basis that the DMMA column pass leaves
    (QD_PREC_FP32, 60, 48, 16, None, 12, 1)])
def test_choice(qdlib, monkeypatch, prec, n1, n2, nth, env, lines, column):
    from qd_b200 import Propagator
    if env:
        monkeypatch.setenv("QD_SLICE_CLUSTER", env)
    d = S.build_case("h+h2", n1, n2, nth, m=nth - 1, total_steps=1, n_energies=5,
                     n_gradient_points=3)
    d.options.precision = prec
    with Propagator(d) as p:
        ch = (C.c_int32 * 4)()
        assert qdlib.qd_kernel_choice(p._h, ch) == 0
    assert list(ch)[:2] == [lines, column]


@pytest.mark.parametrize("fp64,ch,lines,column", [
    (True, [12, 1, 0, 0], "k_axis_f64", "k_column_dmma"),
    (True, [0, 1, 0, 0], "split", "k_column_dmma"),
    (True, [12, 0, 0, 0], "k_axis_f64", "SIMT"),
    (False, [12, 1, 0, 1], "k_axis_f32", "k_column_tc"),
    (False, [0, 0, 0, 1], "split", "SIMT"),
    (False, [10, 1, 1, 1], "4-CTA", "k_column_tc")])
def test_description(fp64, ch, lines, column):
    import bench
    got = bench.describe_choice(ch, fp64)
    assert lines in got["l_space"] and column in got["column"], got


@pytest.mark.gpu
@pytest.mark.parametrize("n1,n2,nth,kinds", [
    (6, 256, 8, (1, 2, 4)),             # 19.1 us a step against 23.6 on the run-time kernels
    (12, 256, 8, (1, 2, 4)),            # 21.2 and 24.3
    (40, 60, 16, (12,)), (96, 240, 8, (12,))])      # 16.8 and 21.2; never timed
def test_grids_of_few_columns_are_timed(qdlib, n1, n2, nth, kinds):
    from qd_b200 import Propagator
    d = S.build_case("h+h2", n1, n2, nth, m=nth - 1, total_steps=1, n_energies=5,
                     n_gradient_points=3)
    d.options.precision = QD_PREC_FP32
    with Propagator(d) as p:
        ch = (C.c_int32 * 4)()
        assert qdlib.qd_kernel_choice(p._h, ch) == 0
    assert ch[0] in kinds
