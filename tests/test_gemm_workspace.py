"""Scratch of split products: each call has its own, made under the stream that the call launches on."""
import threading

import pytest
import torch

from frankentorch_b200.ops import _lib
from frankentorch_b200.ops import kernels as K

FIELDS = [n for n, _ in _lib.FtkGemmDesc._fields_]


class _Library:
    """Stands in for the kernel library: plans two splits for every product that offers a workspace, records launches."""

    def __init__(self, stream):
        self.stream, self.launches, self.plans = stream, [], 0

    def ftk_gemm_plan(self, desc, bn, splits):
        self.plans += 1
        bn._obj.value, splits._obj.value = 128, 2 if desc._obj.workspace else 1
        return 0

    def gemm_packed(self, packed, stream):
        d = _lib.FtkGemmDesc.from_buffer_copy(packed)
        self.launches.append((stream, d.workspace, d.workspace_bytes))
        return 0


@pytest.fixture
def fake(monkeypatch):
    now = [1]                                  # the current stream
    lib = _Library(now)
    made = {}                                  # pointer -> (stream, bytes); tensors are kept, so pointers are distinct
    kept, empty = [], torch.empty

    def recording_empty(*a, **k):
        t = empty(*a, **k)
        kept.append(t)
        made[t.data_ptr()] = (now[0], t.numel() * t.element_size())
        return t

    monkeypatch.setattr(K, "_bf16", lambda t, name: None)
    monkeypatch.setattr(K, "_stream", lambda: now[0])
    monkeypatch.setattr(_lib, "load", lambda *a, **k: lib)
    monkeypatch.setattr(torch, "empty", recording_empty)
    return now, lib, made


def test_products_on_two_streams_do_not_share_scratch(fake):
    now, lib, made = fake
    a, b = torch.zeros(16, 2048, dtype=torch.bfloat16), torch.zeros(24, 2048, dtype=torch.bfloat16)
    for s in (1, 2, 2):
        now[0] = s
        K.gemm(a, b, out_dtype=torch.float32)
    assert [x[0] for x in lib.launches] == [1, 2, 2]
    ptrs = [x[1] for x in lib.launches]
    assert len(set(ptrs)) == 3
    for s, ptr, size in lib.launches:
        assert made[ptr] == (s, 2 * 16 * 24 * 4) and size == 2 * 16 * 24 * 4


def test_scratch_outlives_a_reduction_elsewhere(fake):
    _, lib, made = fake
    a, b = torch.zeros(16, 2048, dtype=torch.bfloat16), torch.zeros(24, 2048, dtype=torch.bfloat16)
    held = []
    K.gemm(a, b, out_dtype=torch.float32, reduce_stream=7, keep=held)
    assert [t.data_ptr() for t in held] == [lib.launches[0][1]]


def test_short_products_neither_plan_nor_allocate(fake):
    _, lib, made = fake
    n = K.SPLIT_ABOVE_K
    a, b = torch.zeros(16, n, dtype=torch.bfloat16), torch.zeros(24, n, dtype=torch.bfloat16)
    out = torch.zeros(16, 24)
    made.clear()
    K.gemm(a, b, out=out)
    assert lib.plans == 0 and not made and lib.launches[0][1:] == (None, 0)


def test_the_planner_never_splits_what_is_not_asked():
    """SPLIT_ABOVE_K against the planner of the library (which runs without a GPU)."""
    import ctypes as C
    lib = _lib.load()
    for M, N, Kd in ((128, 128, K.SPLIT_ABOVE_K), (8, 8, 960), (2048, 128, 896), (128, 128, K.SPLIT_ABOVE_K + 1)):
        for split_k in (0, 2, 4):
            g = _lib.FtkGemmDesc()
            g.M, g.N, g.K, g.L0, g.L1 = M, N, Kd, 1, 1
            g.A = g.B = g.D = g.workspace = 256
            g.workspace_bytes, g.split_k, g.max_ctas = K.GEMM_WORKSPACE_BYTES, split_k, 148
            g.lda = g.ldb = (Kd + 7) // 8 * 8
            g.ldd = N
            bn, sp = C.c_int(0), C.c_int(1)
            assert lib.ftk_gemm_plan(C.byref(g), C.byref(bn), C.byref(sp)) == 0
            assert sp.value == 1 if Kd <= K.SPLIT_ABOVE_K or split_k == 4 else sp.value >= 1


@pytest.mark.gpu
@pytest.mark.parametrize("side", [False, True])
def test_split_products_of_two_threads(cuda_device, side):
    """Two threads, each with a stream (and a reduction stream), split products at the same time: the bits of one alone."""
    g = torch.Generator(device=cuda_device).manual_seed(5)
    probs = [(torch.randn(8192, m, generator=g, device=cuda_device).to(torch.bfloat16),
              torch.randn(8192, n, generator=g, device=cuda_device).to(torch.bfloat16)) for m, n in ((768, 768), (512, 1024))]
    call = lambda dy, x, **k: K.gemm(dy, x, a_mn=True, b_mn=True, out_dtype=torch.float32, split_k=4, **k)   # noqa: E731
    refs = [call(*p) for p in probs]
    torch.cuda.synchronize()
    bad = [0, 0]

    def work(i):
        with torch.cuda.device(cuda_device):
            main, aside = torch.cuda.Stream(), torch.cuda.Stream()
            with torch.cuda.stream(main):
                for _ in range(60):
                    out = call(*probs[i], reduce_stream=aside.cuda_stream) if side else call(*probs[i])
                    main.wait_stream(aside)
                    if not torch.equal(out, refs[i]):
                        bad[i] += 1
    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    K.check_status()
    assert bad == [0, 0]
