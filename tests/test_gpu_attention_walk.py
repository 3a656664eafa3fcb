"""Attention kernels with fewer and with more work items than SMs, at the edges of their 128-row blocks: gradients and
outputs against 64-bit arithmetic, and the same bits again on a second run."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, go, causal):
    q, k, v = (t.double().detach().requires_grad_(True) for t in (q, k, v))
    S = q.shape[1]
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) / math.sqrt(q.shape[-1])
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1), -math.inf)
    o = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v)
    return (o.detach(),) + torch.autograd.grad(o, (q, k, v), go.double())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H", [
    (1, 1, 1), (1, 127, 1), (2, 128, 3), (1, 129, 2), (1, 257, 1),
    (3, 383, 5),        # three blocks, ragged
    (2, 640, 16),       # 160 items: a second round with a few items only
    (5, 264, 40),       # 600 items, several rounds, one or two blocks each
    (1, 1500, 3),       # twelve blocks, ragged
])
def test_walk_over_items(cuda_device, B, S, H, hd, causal):
    from frankentorch_b200.ops import kernels as K
    g = torch.Generator().manual_seed(B * 1000 + S)
    qkv = torch.randn(B, S, 3, H, hd, generator=g).to(torch.bfloat16).to(cuda_device)
    q, k, v = (qkv[:, :, i] for i in range(3))
    go = torch.randn(B, S, H, hd, generator=g).to(torch.bfloat16).to(cuda_device)
    runs = []
    for _ in range(2):
        o, lse = K.attention_fwd(q, k, v, causal=causal)
        d = torch.full_like(qkv, float("nan"))
        K.attention_bwd(q, k, v, o, lse, go, causal=causal, dq=d[:, :, 0], dk=d[:, :, 1], dv=d[:, :, 2])
        runs.append((o, d))
    K.check_status()
    assert torch.equal(runs[0][0], runs[1][0]) and torch.equal(runs[0][1], runs[1][1])
    o, d = runs[0]
    ro, rq, rk, rv = _reference(q, k, v, go, causal)
    # P, dS and the outputs are rounded to bf16 (2^-9 each, independent over the sums): under 1 % of the 2-norm
    for name, got, ref in (("o", o, ro), ("dq", d[:, :, 0], rq), ("dk", d[:, :, 1], rk), ("dv", d[:, :, 2], rv)):
        assert got.isfinite().all(), name
        err = float((got.double() - ref).norm() / ref.norm().clamp_min(1e-3 * go.double().norm()))
        assert err < 1e-2, (name, err)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H", [(8, 256, 40), (8, 200, 40), (4, 300, 80), (16, 128, 40)])
def test_short_items_in_turns(cuda_device, B, S, H, causal):
    """Several items of one or two key blocks per CTA, where the softmax groups of head size 64 meet only in the turn order:
    the same bits on every run, no abandoned wait, the values of 64-bit arithmetic."""
    from frankentorch_b200.ops import kernels as K
    g = torch.Generator().manual_seed(S)
    qkv = torch.randn(B, S, 3, H, 64, generator=g).to(torch.bfloat16).to(cuda_device)
    q, k, v = (qkv[:, :, i] for i in range(3))
    first, _ = K.attention_fwd(q, k, v, causal=causal)
    for _ in range(40):
        again, _ = K.attention_fwd(q, k, v, causal=causal)
        assert torch.equal(again, first)
    K.check_status()
    ref = _reference(q, k, v, torch.zeros_like(first), causal)[0]
    assert float((first.double() - ref).norm()) < 1e-2 * float(ref.norm())      # P and the output are rounded to bf16


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H", [(8, 100, 40), (6, 250, 40), (4, 300, 60), (3, 520, 50)])
def test_backward_of_short_items(cuda_device, B, S, H, hd, causal):
    """Several items of one to five blocks per CTA, whose outputs leave while the next item runs, through tiles that are loaded
    again: the same bits on every run, the values of 64-bit arithmetic, nothing written beside ragged rows and columns."""
    from frankentorch_b200.ops import kernels as K
    g = torch.Generator(device=cuda_device).manual_seed(S + hd)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda_device).to(torch.bfloat16)      # noqa: E731
    pad = 16                                           # columns of each row that belong to nobody
    store = rnd(B, S + 1, 3 * H * hd + pad)            # and a row behind every sequence
    view = lambda t: [t[:, :S, i * H * hd:(i + 1) * H * hd].unflatten(-1, (H, hd)) for i in range(3)]      # noqa: E731
    q, k, v = view(store)
    go = rnd(B, S, H, hd)
    o, lse = K.attention_fwd(q, k, v, causal=causal)
    first = None
    for _ in range(8):
        d = torch.full_like(store, 7.0)
        dq, dk, dv = view(d)
        K.attention_bwd(q, k, v, o, lse, go, causal=causal, dq=dq, dk=dk, dv=dv)
        first = d if first is None else first
        assert torch.equal(first, d)
    K.check_status()
    assert bool((first[:, S] == 7.0).all()) and bool((first[:, :, -pad:] == 7.0).all())
    for got, ref in zip(view(first), _reference(q, k, v, go, causal)[1:]):
        assert got.isfinite().all()
        assert float((got.double() - ref).norm() / ref.norm()) < 1e-2      # as above


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,S,H,strides", [
    (1, 200, 3, lambda S, H, hd: (S * H * hd + 1, H * hd, hd, 1)),      # one sequence of a buffer with an odd row
    (1, 1, 5, lambda S, H, hd: (3, 7, hd, 1)),                          # one token: neither stride is stepped over
    (1, 70, 1, lambda S, H, hd: (5, hd, 3, 1)),                         # one head
    (1, 1, 1, lambda S, H, hd: (1, 1, 1, 1)),
    (2, 130, 1, lambda S, H, hd: (S * hd, hd, 1, 1)),
    (3, 1, 2, lambda S, H, hd: (2 * hd, 1, hd, 1)),
])
def test_output_strides_of_extents_of_one(cuda_device, B, S, H, strides, hd):
    """A stride that nothing steps over may be anything, also one that is no multiple of 16 bytes."""
    from frankentorch_b200.ops import kernels as K
    g = torch.Generator(device=cuda_device).manual_seed(5)
    q, k, v = (torch.randn(B, S, H, hd, generator=g, device=cuda_device).to(torch.bfloat16) for _ in range(3))
    ref, ref_lse = K.attention_fwd(q, k, v, causal=True)
    store = torch.full((B * S * H * hd + 64,), 7.0, dtype=torch.bfloat16, device=cuda_device)
    out, lse = K.attention_fwd(q, k, v, causal=True, out=store.as_strided((B, S, H, hd), strides(S, H, hd)))
    K.check_status()
    assert torch.equal(out, ref) and torch.equal(lse, ref_lse)
    assert bool((store[B * S * H * hd:] == 7.0).all())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,S,H,causal", [
    (4, 100, 37, True),        # 148 items: one for each CTA
    (1, 64, 149, False),       # one item more, of one block
    (1, 1920, 10, True),       # 150 items of up to fifteen blocks: a second item is seldom
    (1, 2100, 12, False),      # 204 items of seventeen blocks: outputs leave at the end of their item
    (2, 700, 31, True),        # 372 items of up to six blocks: under the next one
])
def test_forms_of_the_backward(cuda_device, B, S, H, causal, hd):
    """Which form of the kernels runs follows from the number of items and of blocks; values as in the walk over items."""
    test_walk_over_items(cuda_device, B=B, S=S, H=H, hd=hd, causal=causal)
