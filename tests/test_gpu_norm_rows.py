"""Norm kernels at the widths where the split of a row over lanes and warps changes, with fewer rows than a step and with
several steps per block: values, gradients and column sums against 64-bit arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu

COLS = [8, 256, 264, 512, 768, 776, 1024, 1536, 1544, 2048, 3072, 3080, 4096, 4104, 6144, 6152, 8192, 8200,
        16384, 16392, 20008]


def _norm(x, g, b, rms, eps):
    if rms:
        return x * torch.rsqrt((x ** 2).mean(-1, keepdim=True) + eps) * g
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), g, b, eps)


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows", [1, 7, 700, 5003])
@pytest.mark.parametrize("cols", COLS)
def test_norm(cuda_device, rows, cols, rms, most=12_000_000):
    from frankentorch_b200.ops import kernels as K
    if rows * cols > most:
        rows = most // cols
    gen = torch.Generator(device=cuda_device).manual_seed(cols + rows)
    rnd = lambda *s, sc=1.0, m=0.0: (torch.randn(*s, generator=gen, device=cuda_device) * sc + m).to(torch.bfloat16)   # noqa: E731
    x, dy, add = rnd(rows, cols, sc=2.0, m=0.3), rnd(rows, cols), rnd(rows, cols)
    g, b = rnd(cols, sc=0.1, m=1.0), rnd(cols, sc=0.1)
    xd, gd, bd = (t.double().requires_grad_(True) for t in (x, g, b))
    eps = 1e-5
    y = _norm(xd, gd, bd, rms, eps)
    refs = torch.autograd.grad(y, (xd, gd) if rms else (xd, gd, bd), dy.double())

    def close(got, ref, tol):
        assert got.isfinite().all()
        assert float((got.double() - ref).norm()) <= tol * float(ref.norm()) + 1e-6

    bf16 = 2.0 ** -8                    # one rounding to bf16, 2^-9 relative at most
    f32 = 3e-6 * max(1.0, rows ** 0.5 / 16)      # fp32 sums over the rows in a fixed order, rounding errors of random sign
    if rms:
        got, rstd = K.rmsnorm_fwd(x, g, eps)
        dx, dg = K.rmsnorm_bwd(dy, x, g, rstd)
        pre = torch.ones(cols, device=cuda_device)
        K.rmsnorm_bwd(dy, x, g, rstd, dgamma=pre, accumulate=True)
        close(pre, refs[1] + 1, f32)
    else:
        got, mean, rstd, _ = K.layernorm_fwd(x, g, b, eps)
        dx, dg, db = K.layernorm_bwd(dy, x, g, mean, rstd)
        close(db, refs[2], f32)
        dx2, dg2, db2 = K.layernorm_bwd(dy, x, g, mean, rstd, dx_add=add)
        close(dx2, refs[0] + add.double(), bf16)
        assert torch.equal(dg, dg2) and torch.equal(db, db2)
        # residual form of the forward: statistics of the rounded sum
        y2, m2, r2, xs = K.layernorm_fwd(x, g, b, eps, resid=add)
        assert torch.equal(xs, (x.float() + add.float()).to(torch.bfloat16))
        close(y2, _norm(xs.double(), gd.detach(), bd.detach(), False, eps), bf16)
    K.check_status()
    close(got, y.detach(), bf16)
    close(dx, refs[0], bf16)
    close(dg, refs[1], f32)


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,cols", [
    (23999, 64), (24000, 64), (24000, 128), (24000, 136), (24000, 256), (24000, 264), (131073, 256),     # separate backward passes
    (4095, 1024), (4096, 1024), (499, 1544), (500, 1544), (8191, 2048), (8192, 2048),                   # warps per row, forward
])
def test_norm_where_the_number_of_rows_decides(cuda_device, rows, cols, rms):
    """Both sides of the rules that look at the number of rows."""
    test_norm(cuda_device, rows, cols, rms, most=1 << 26)


@pytest.mark.parametrize("rows,cols", [
    (1, 2), (64, 130), (512, 96), (513, 96),       # up to and beyond eight row blocks of 64: another number of groups
    (1537, 4104), (8192, 40), (8193, 40),          # two rounds of loads, 128 and 129 blocks
    (8200, 8184), (8200, 8192),                    # the width from which the wide form stays
    (300, 34), (3000, 1026),                       # rows that are not whole 16-byte segments: blocks of 256 rows
])
def test_column_sums(cuda_device, rows, cols):
    from frankentorch_b200.ops import kernels as K
    x = torch.randn(rows, cols, generator=torch.Generator(device=cuda_device).manual_seed(rows), device=cuda_device).to(torch.bfloat16)
    ref = x.double().sum(0)
    bound = 2.0 ** -24 * (8 + rows ** 0.5) * x.double().abs().sum(0) + 1e-6     # rounding errors of random sign, fp32 sums
    out = K.colsum(x)
    assert bool(((out.double() - ref).abs() <= bound).all())
    pre = torch.full((cols,), 2.0, device=cuda_device)
    K.colsum(x, out=pre, accumulate=True)
    assert torch.equal(pre, out + 2.0)
    assert torch.equal(K.colsum(x), out)
