"""Every tile width of the GEMM (single CTA 128 / 192 / 256, CTA pair 256 x 128 / 192 / 256) with every epilogue
instantiation at the edges of its tiles, with both operands given [K, rows], with split reductions (also such that leave the
last split empty), and the general path of outputs without aligned 16-byte segments."""
import pytest
import torch

pytestmark = pytest.mark.gpu

WIDTHS = [128, 192, 256, 256 + 128, 256 + 192, 256 + 256]


def _rand(shape, seed, dev, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).to(dev)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _dgelu(x):
    x = x.clone().requires_grad_(True)
    return torch.autograd.grad(_gelu(x).sum(), x)[0]


def _close(out, ref, act=False):
    # the output's rounding (at most 2^-9 relative for bf16, twice that here), the error of fp32 sums of at most 1096
    # products whose squares add up to about one (1096 * 2^-24 = 7e-5), and 2^-10 |x| of the hardware tanh
    bound = (2.0 ** -8 if out.dtype == torch.bfloat16 else 2.0 ** -20) * ref.abs() + 1e-4
    if act:
        bound = bound + 2.0 ** -9 * ref.abs().max()
    assert out.double().isfinite().all()
    err = (out.double() - ref).abs()
    assert bool((err <= bound).all()), float((err - bound).max())


@pytest.mark.parametrize("bn", WIDTHS)
@pytest.mark.parametrize("M,N,K", [
    (256, 64, 64),          # one tile, one k-block, columns end inside the tile
    (1, 8, 8),              # the smallest extents
    (257, 200, 136),        # one row into the second pair tile, ragged N and K
    (384, 584, 1096),       # several tiles, more k-blocks than stages
])
@pytest.mark.parametrize("kind", ["plain", "bias", "bias_resid", "gelu", "gelu_aux", "dgelu", "relu_resid", "f32", "f32_acc"])
def test_tiles_and_epilogues(cuda_device, bn, M, N, K, kind):
    from frankentorch_b200.ops import kernels as k
    b_mn = kind in ("dgelu", "plain")            # the layouts that training uses: dgrad reads the weight as [K, N]
    a, w = _rand((M, K), 1, cuda_device), _rand((K, N) if b_mn else (N, K), 2, cuda_device, K ** -0.5)
    bias, r = _rand((N,), 3, cuda_device), _rand((M, N), 4, cuda_device)
    ref = a.double() @ (w.double() if b_mn else w.double().t())
    kw, aux = {}, None
    if kind in ("bias", "bias_resid", "gelu", "gelu_aux", "relu_resid"):
        kw["bias"], ref = bias, ref + bias.double()
    if kind.startswith("gelu"):
        pre, ref = ref, _gelu(ref)
        kw["epi"] = k.EPI_GELU_TANH
        if kind == "gelu_aux":
            kw["aux"] = aux = torch.empty((M, N), dtype=torch.bfloat16, device=cuda_device)
    if kind == "dgelu":
        ref = ref * _dgelu(r.double())
        kw.update(epi=k.EPI_MUL_DGELU_TANH, resid=r)
    if kind == "relu_resid":
        kw["epi"], ref = k.EPI_RELU, torch.relu(ref)
    if kind in ("bias_resid", "relu_resid"):
        kw["resid"], ref = r, ref + r.double()
    if kind.startswith("f32"):
        kw.update(out_dtype=torch.float32, split_k=1)
        if kind == "f32_acc":
            out0 = torch.full((M, N), 0.5, device=cuda_device)
            kw.update(out=out0, accumulate=True)
            ref = ref + 0.5
    out = k.gemm(a, w, b_mn=b_mn, force_bn=bn, **kw)
    k.check_status()
    _close(out, ref, act="gelu" in kind)
    if aux is not None:
        _close(aux, pre)


@pytest.mark.parametrize("bn", WIDTHS)
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (264, 200, 136), (384, 584, 1096), (520, 264, 72)])
def test_weight_gradient_form(cuda_device, bn, M, N, K, accumulate):
    """Both operands [K, rows], fp32 output: what a weight gradient runs."""
    from frankentorch_b200.ops import kernels as k
    a, b = _rand((K, M), 11, cuda_device), _rand((K, N), 12, cuda_device, K ** -0.5)
    ref = a.double().t() @ b.double()
    out = torch.full((M, N), 0.5 if accumulate else float("nan"), device=cuda_device)
    k.gemm(a, b, a_mn=True, b_mn=True, out=out, accumulate=accumulate, force_bn=bn, split_k=1)
    k.check_status()
    _close(out, ref + 0.5 if accumulate else ref)


@pytest.mark.parametrize("bn", WIDTHS)
@pytest.mark.parametrize("form", ["nt", "tn", "bf16_acc"])
@pytest.mark.parametrize("splits,K", [
    (2, 1024),            # the shortest that may be split: eight k-blocks each
    (3, 1600),            # 25 k-blocks: 9, 9 and 7
    (12, 6200),           # 97 k-blocks, nine each: the twelfth split has none
])
def test_split_reductions(cuda_device, bn, form, splits, K):
    from frankentorch_b200.ops import kernels as k
    M, N = 264, 200
    mn = form == "tn"
    a, b = _rand((K, M) if mn else (M, K), 13, cuda_device), _rand((K, N) if mn else (N, K), 14, cuda_device, K ** -0.5)
    ref = a.double().t() @ b.double() if mn else a.double() @ b.double().t()
    out = torch.full((M, N), 0.25, dtype=torch.bfloat16 if form == "bf16_acc" else torch.float32, device=cuda_device)
    kw = dict(a_mn=mn, b_mn=mn, force_bn=bn, split_k=splits)
    k.trace_begin()
    k.gemm(a, b, out=out, accumulate=form != "nt", **kw)
    name, = k.trace_end()
    assert name.endswith("splitK=%d>" % splits)
    k.check_status()
    if form != "nt":
        ref = ref + 0.25
    # as _close, with fp32 sums of K products (6200 * 2^-24 at most) and the bf16 output's rounding
    bound = (2.0 ** -8 if out.dtype == torch.bfloat16 else 2.0 ** -20) * ref.abs() + 4e-4
    assert bool(((out.double() - ref).abs() <= bound).all())
    again = torch.full_like(out, 0.25)
    k.gemm(a, b, out=again, accumulate=form != "nt", **kw)
    assert torch.equal(again, out)


@pytest.mark.parametrize("bn", WIDTHS)
@pytest.mark.parametrize("N,ldd,off", [(37, 37, 0), (40, 41, 0), (40, 40, 1), (72, 80, 3)])
def test_rows_without_aligned_segments(cuda_device, bn, N, ldd, off):
    """Odd widths, leading dimensions and bases, bf16 accumulation: the general epilogue, nothing written beside it."""
    from frankentorch_b200.ops import kernels as k
    M, K = 200, 72
    a, w = _rand((M, K), 5, cuda_device), _rand((N, K), 6, cuda_device, K ** -0.5)
    bias = _rand((N,), 7, cuda_device)
    store = torch.full((M * ldd + off + 8,), 7.0, dtype=torch.bfloat16, device=cuda_device)
    out = store[off:off + M * ldd].view(M, ldd)[:, :N]
    k.gemm(a, w, bias=bias, out=out, force_bn=bn)
    ref = a.double() @ w.double().t() + bias.double()
    _close(out, ref)
    k.gemm(a, w, out=out, accumulate=True, force_bn=bn)
    k.check_status()
    assert float((out.double() - (2 * ref - bias.double())).abs().max()) <= 2.0 ** -7 * float(ref.abs().max()) + 1e-3
    mask = torch.ones_like(store, dtype=torch.bool)
    mask[off:off + M * ldd].view(M, ldd)[:, :N] = False
    assert bool((store[mask] == 7.0).all())


@pytest.mark.parametrize("bn", WIDTHS)
@pytest.mark.parametrize("kind", ["plain", "bias_gelu", "relu_resid", "dgelu"])
@pytest.mark.parametrize("ldr", [72, 73, 76])
def test_bf16_accumulation_and_residual_rows(cuda_device, bn, kind, ldr):
    """A bf16 output that is added to, with an operand whose rows are whole 16-byte segments (72), 2 or 8 bytes off them."""
    from frankentorch_b200.ops import kernels as k
    M, N, K = 333, 72, 136
    a, w, bias = _rand((M, K), 31, cuda_device), _rand((N, K), 32, cuda_device, K ** -0.5), _rand((N,), 33, cuda_device)
    out, r = _rand((M, N), 34, cuda_device), _rand((M, ldr), 35, cuda_device)[:, :N]
    ref, kw = a.double() @ w.double().t(), {}
    if kind == "bias_gelu":
        ref, kw = _gelu(ref + bias.double()), {"bias": bias, "epi": k.EPI_GELU_TANH}
    elif kind == "relu_resid":
        ref, kw = torch.relu(ref) + r.double(), {"epi": k.EPI_RELU, "resid": r}
    elif kind == "dgelu":
        ref, kw = ref * _dgelu(r.double()), {"epi": k.EPI_MUL_DGELU_TANH, "resid": r}
    fresh = k.gemm(a, w, force_bn=bn, split_k=1, **kw)
    ref_acc = ref + out.double()
    k.gemm(a, w, out=out, accumulate=True, force_bn=bn, split_k=1, **kw)
    k.check_status()
    _close(fresh, ref, act="gelu" in kind)
    _close(out, ref_acc, act="gelu" in kind)


def test_grouped_products_with_unaligned_outputs(cuda_device):
    from frankentorch_b200.ops import kernels as k
    K, shapes = 264, [(264, 200), (16, 8), (520, 40)]
    probs, refs = [], []
    for i, (M, N) in enumerate(shapes):
        a, b = _rand((K, M), 10 + i, cuda_device), _rand((K, N), 20 + i, cuda_device, K ** -0.5)
        out = torch.full((M, N + 1), 0.25, device=cuda_device)[:, :N]
        probs.append((a, b, out, True))
        refs.append(a.double().t() @ b.double() + 0.25)
    k.gemm_grouped(probs)
    k.check_status()
    for (_, _, out, _), ref in zip(probs, refs):
        _close(out, ref)


@pytest.mark.parametrize("bn", [256 + 128, 256 + 192, 256 + 256])
@pytest.mark.parametrize("M,N,K", [
    (4 * 256 + 8, 264, 32768),        # five row blocks of a large A in groups of four: a last group of one
    (7 * 256, 8 * 256 + 136, 24576),  # more column blocks, a last group of three
    (10 * 256 + 136, 17 * 256, 13312),  # groups of eight where the column blocks are many
])
@pytest.mark.parametrize("splits", [1, 3])
def test_row_block_groups(cuda_device, bn, M, N, K, splits):
    """An A beyond half of L2 is walked in groups of row blocks: every tile once, also with a last group that is not whole."""
    from frankentorch_b200.ops import kernels as k
    assert 2 * M * K > 64 << 20
    a, w = _rand((M, K), 21, cuda_device), _rand((N, K), 22, cuda_device, K ** -0.5)
    ref = a.double() @ w.double().t()
    out = torch.full((M, N), float("nan"), device=cuda_device)
    k.gemm(a, w, out=out, force_bn=bn, split_k=splits)
    k.check_status()
    # fp32 sums of K products whose squares add up to about one: at most K * 2^-24 of them, 2e-3
    assert float((out.double() - ref).abs().max()) <= K * 2.0 ** -24


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("mn", [True, False])
def test_wide_grouped_tiles(cuda_device, pad, accumulate, mn):
    """Groups with long reductions on few CTAs take 256 x 384 tiles: several per pair, ragged rows, columns and k-blocks."""
    from frankentorch_b200.ops import kernels as k
    K, shapes = 4104, [(264, 384), (520, 760), (256, 392)]
    probs, refs = [], []
    for i, (M, N) in enumerate(shapes):
        a, b = _rand((K, M), 30 + i, cuda_device), _rand((K, N), 40 + i, cuda_device, K ** -0.5)
        if not mn:
            a, b = a.t().contiguous(), b.t().contiguous()
        out = torch.full((M, N + pad), 0.25 if accumulate else float("nan"), device=cuda_device)[:, :N]
        probs.append((a, b, out, accumulate))
        refs.append((a.double().t() @ b.double() if mn else a.double() @ b.double().t()) + (0.25 if accumulate else 0.0))
    for ctas in (4, 0):
        for _, _, out, _ in probs:
            out.fill_(0.25)
        k.gemm_grouped(probs, a_mn=mn, b_mn=mn, max_ctas=ctas)
        k.check_status()
        for (_, _, out, _), ref in zip(probs, refs):
            # fp32 sums of K products whose squares add up to about one
            assert float((out.double() - ref).abs().max()) <= K * 2.0 ** -24 + 2.0 ** -20 * float(ref.abs().max())


@pytest.mark.parametrize("bn", [256 + 160, 256 + 224])
@pytest.mark.parametrize("M,N,K", [(256, 64, 64), (257, 200, 136), (384, 584, 1096), (512, 160, 72), (300, 232, 64)])
@pytest.mark.parametrize("kind", ["plain", "bias_resid", "gelu_aux", "dgelu", "relu_resid", "f32_acc"])
def test_widths_of_an_odd_number_of_chunks(cuda_device, bn, M, N, K, kind):
    """Pair tiles of 160 and 224 columns: the two warps of a lane quarter drain unequal shares."""
    test_tiles_and_epilogues(cuda_device, bn=bn, M=M, N=N, K=K, kind=kind)


@pytest.mark.parametrize("bn", [256 + 160, 256 + 224])
def test_widths_of_an_odd_number_of_chunks_other_forms(cuda_device, bn):
    for M, N, K in ((264, 200, 136), (384, 584, 1096)):
        test_weight_gradient_form(cuda_device, bn=bn, accumulate=True, M=M, N=N, K=K)
    test_split_reductions(cuda_device, bn=bn, form="tn", splits=3, K=1600)
    test_rows_without_aligned_segments(cuda_device, bn=bn, N=37, ldd=37, off=0)
    test_bf16_accumulation_and_residual_rows(cuda_device, bn=bn, kind="bias_gelu", ldr=73)
    test_row_block_groups(cuda_device, bn=bn, M=7 * 256, N=8 * 256 + 136, K=24576, splits=1)


@pytest.mark.parametrize("bn", [256 + 160, 256 + 256])
@pytest.mark.parametrize("M,N,K", [
    (17 * 256 + 8, 8200, 8200),       # groups of sixteen for a B beyond L2, a last group of two
    (22 * 256 + 136, 4352, 6144),     # groups of eight, a last group of seven
])
def test_row_block_groups_of_a_large_b(cuda_device, bn, M, N, K):
    test_row_block_groups(cuda_device, bn=bn, M=M, N=N, K=K, splits=1)


@pytest.mark.parametrize("mn", [True, False])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("pad", [4, 1])
@pytest.mark.parametrize("K,ctas,width", [(4104, 4, 384), (4104, 0, 192), (136, 2, 192), (8200, 2, 384)])
def test_both_widths_of_grouped_tiles(cuda_device, K, ctas, width, pad, accumulate, mn):
    """The width that the case is meant for runs, and nothing is written beside the outputs, nor is anything of them left out."""
    from frankentorch_b200.ops import kernels as k
    probs, refs, stores = [], [], []
    for i, (M, N) in enumerate([(264, 384), (520, 760), (256, 392), (304, 376)]):
        a, b = _rand((K, M), 50 + i, cuda_device), _rand((K, N), 60 + i, cuda_device, K ** -0.5)
        ref = a.double().t() @ b.double()
        if not mn:
            a, b = a.t().contiguous(), b.t().contiguous()
        store = torch.full((M + 1, N + pad), 0.25, device=cuda_device)
        if not accumulate:
            store[:M, :N] = float("nan")
        probs.append((a, b, store[:M, :N], accumulate))
        refs.append(ref + 0.25 if accumulate else ref)
        stores.append(store)
    k.trace_begin()
    k.gemm_grouped(probs, a_mn=mn, b_mn=mn, max_ctas=ctas)
    assert k.trace_end() == ["ftk::gemm_group_bf16_sm100<256x%d,cta_group2,problems=4>" % width]
    k.check_status()
    for store, ref in zip(stores, refs):
        M, N = ref.shape
        assert bool((store[M:] == 0.25).all()) and bool((store[:, N:] == 0.25).all())
        # fp32 sums of K products whose squares add up to about one
        assert float((store[:M, :N].double() - ref).abs().max()) <= K * 2.0 ** -24 + 2.0 ** -20 * float(ref.abs().max())
