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
    """Operands whose rows are not whole 128-byte lines pay more per k-block, so their products are split where the aligned ones
    of the same tiles are not: 2136 x 632 over 12874 rows took 73 us in 45 tiles and 51 us in eight splits, 1500 x 1000 x 5000
    30 us in 48 tiles and 22 us in three splits, 1500 x 1024 x 5056 17.7 us unsplit and 18.8 in three."""
    assert _plan(2136, 632, 12874, a_mn=1, b_mn=1, f32=1)[2] > 1
    assert _plan(2176, 640, 8192, a_mn=1, b_mn=1, f32=1)[2] == 1
    assert _plan(1500, 1000, 5000, b_mn=1)[2] > 1 and _plan(1500, 1024, 5056, b_mn=1)[2] == 1


@pytest.mark.parametrize("bn", [384, 448, 512])
def test_a_pair_tile_that_cannot_run_is_refused(bn):
    assert _plan(256, 256, 64, force_bn=bn)[:2] == (0, bn)
    assert _plan(256, 256, 64, force_bn=bn, max_ctas=2)[:2] == (0, bn)
    assert _plan(256, 256, 64, force_bn=bn, max_ctas=1)[0] == -5
    g = _desc(256, 256, 64, force_bn=bn)
    g.seg_counts, g.seg_rows = 256, 128
    out = C.c_int(0), C.c_int(1)
    assert _lib.load().ftk_gemm_plan(C.byref(g), C.byref(out[0]), C.byref(out[1])) == -5


@pytest.mark.parametrize("max_ctas", [1, 2, 3, 36, 37, 148])
@pytest.mark.parametrize("shapes", [[(64, 64)], [(2304, 768), (768, 768), (3072, 768), (768, 3072)]])
def test_a_group_keeps_to_its_ctas(shapes, max_ctas):
    fn = _lib.load().ftk_gemm_group_ctas
    fn.argtypes, fn.restype = [C.POINTER(_lib.FtkGemmDesc), C.c_int], C.c_int
    arr = (_lib.FtkGemmDesc * len(shapes))(*[_desc(m, n, 512, a_mn=1, b_mn=1, f32=1, max_ctas=max_ctas) for m, n in shapes])
    ctas = fn(arr, len(shapes))
    assert 1 <= ctas <= max_ctas and (ctas == 1) == (max_ctas == 1)


def test_widths_that_fill_the_last_wave():
    """1500 x 5120 x 1280 is 138 tiles of 256 x 224 on 74 pairs, 1500 x 3840 x 1280 144 of 256 x 160; a B given [K, N] loads whole
    64-column boxes, so these widths are left out there."""
    assert _plan(1500, 5120, 1280)[:2] == (0, 480) and _plan(1500, 3840, 1280)[:2] == (0, 416)
    assert _plan(1500, 5120, 1280, b_mn=1)[1] not in (416, 480) and _plan(1500, 3840, 1280, b_mn=1)[1] not in (416, 480)
    assert _plan(8192, 2304, 768)[:2] == (0, 512) and _plan(8192, 3072, 768)[:2] == (0, 448)


@pytest.mark.parametrize("M,N,K,rows", [
    (4096, 8192, 8192, 16),        # A is half of L2: m fastest over its 16 row blocks
    (8192, 2048, 8192, 4), (16384, 8192, 4096, 8), (8192, 8192, 8192, 8),      # B within L2: it is read again from there
    (8192, 8448, 8192, 16), (16384, 32768, 4096, 16), (8192, 50304, 8192, 16),      # B beyond L2: fewer passes over it
    (6144, 12288, 8192, 16), (6144, 50304, 8192, 24), (4096, 24576, 16384, 16),      # several times L2, few row blocks: one pass
])
def test_row_block_groups_follow_both_operands(M, N, K, rows):
    """A B beyond L2 is read from memory again for every group: groups of 8 took 8 % longer than none for 6144 x 50304 x 8192, 5 % for
    8192 x 50304 x 8192."""
    for b_mn in (0, 1):
        assert _plan(M, N, K, b_mn=b_mn)[:2] == (0, 512)
        assert _lib.load().ftk_gemm_walk(C.byref(_desc(M, N, K, b_mn=b_mn))) == rows
    assert _lib.load().ftk_gemm_walk(C.byref(_desc(64, N, K))) == 0
    assert _lib.load().ftk_gemm_walk(C.byref(_desc(0, N, K))) == -2


def test_wide_tiles_of_a_group():
    """256 x 384 tiles where they fill the pairs and the reduction is long: the weight gradients of a block of 768 are 72 of them
    (144 CTAs) over 8192 rows, and 144 narrow ones on all CTAs over 512."""
    fn = _lib.load().ftk_gemm_group_ctas
    fn.argtypes, fn.restype = [C.POINTER(_lib.FtkGemmDesc), C.c_int], C.c_int
    for rows, ctas in ((8192, 144), (512, 148)):
        shapes = [(2304, 768), (768, 768), (3072, 768), (768, 3072)]
        arr = (_lib.FtkGemmDesc * 4)(*[_desc(m, n, rows, a_mn=1, b_mn=1, f32=1) for m, n in shapes])
        assert fn(arr, 4) == ctas


def test_the_width_of_a_group_is_reported(monkeypatch):
    """The trace of a grouped launch names the tile that the planner picks."""
    import torch
    from frankentorch_b200.ops import kernels as K
    lib = _lib.load()

    class Library:
        def ftk_gemm_group_bf16(self, arr, n, stream):
            return 0

        def ftk_gemm_group_width(self, arr, n):
            return lib.ftk_gemm_group_width(arr, n)

    monkeypatch.setattr(K, "_bf16", lambda t, name: None)
    monkeypatch.setattr(K, "_stream", lambda: 0)
    monkeypatch.setattr(_lib, "load", lambda *a, **k: Library())
    names = []
    for rows, ctas in ((8192, 148), (512, 148), (8192, 1)):
        probs = [(torch.empty(rows, m, dtype=torch.bfloat16), torch.empty(rows, n, dtype=torch.bfloat16), torch.empty(m, n), False)
                 for m, n in ((2304, 768), (768, 768), (3072, 768), (768, 3072))]
        K.trace_begin()
        K.gemm_grouped(probs, max_ctas=ctas)
        names += K.trace_end()
    assert names == ["ftk::gemm_group_bf16_sm100<256x384,cta_group2,problems=4>",
                     "ftk::gemm_group_bf16_sm100<256x192,cta_group2,problems=4>", "ftk::gemm_bf16_sm100<128x192,problems=4>"]
    assert lib.ftk_gemm_group_width(None, 1) == -2


@pytest.mark.gpu
def test_a_group_on_one_cta(cuda_device):
    import torch
    from frankentorch_b200.ops import kernels as K
    g = torch.Generator(device=cuda_device).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda_device).to(torch.bfloat16)      # noqa: E731
    probs = [(rnd(264, m), rnd(264, n)) for m, n in ((264, 200), (16, 8), (520, 40))]
    outs = []
    for max_ctas in (0, 1):
        o = [torch.full((a.shape[1], b.shape[1]), 0.25, device=cuda_device) for a, b in probs]
        K.gemm_grouped([(a, b, t, True) for (a, b), t in zip(probs, o)], max_ctas=max_ctas)
        outs.append(o)
    K.check_status()
    assert all(torch.equal(x, y) for x, y in zip(*outs))
