"""Tile planner of the GEMM (host code, runs without a GPU)."""
import ctypes as C

import pytest

from frankentorch_b200.ops import _lib


def _desc(M, N, K, *, a_mn=0, b_mn=0, f32=0, max_ctas=148, force_bn=0, split_k=0, workspace=64 << 20):
    g = _lib.FtkGemmDesc()
    g.M, g.N, g.K, g.L0, g.L1, g.a_mn, g.b_mn = M, N, K, 1, 1, a_mn, b_mn
    g.A = g.B = g.D = g.workspace = 256          # aligned stand-ins: the planner looks at extents and alignment
    g.workspace_bytes = workspace
    g.lda, g.ldb = ((M if a_mn else K) + 7) // 8 * 8, ((N if b_mn else K) + 7) // 8 * 8
    g.ldd, g.out_fp32, g.max_ctas, g.force_bn, g.split_k = N, f32, max_ctas, force_bn, split_k
    return g


def _plan(*a, **k):
    bn, sp = C.c_int(0), C.c_int(1)
    rc = _lib.load().ftk_gemm_plan(C.byref(_desc(*a, **k)), C.byref(bn), C.byref(sp))
    return rc, bn.value, sp.value


def test_rows_off_the_lines_are_charged():
    """A weight gradient of operands whose rows are not whole 128-byte lines pays more per k-block, so it is split where the
    aligned one of the same tiles is not: 45 tiles of 256 x 128 on 74 pairs took 73 us, two splits of 256 x 192 53 us."""
    assert _plan(2136, 632, 12874, a_mn=1, b_mn=1, f32=1) == (0, 448, 2)
    assert _plan(2176, 640, 8192, a_mn=1, b_mn=1, f32=1)[2] == 1
    # the charge is for operands given [K, rows] alone
    assert _plan(2136, 632, 2000)[1:] == _plan(2136, 632, 2048)[1:]
