"""Kernels that follow one another, with grids at and beyond the limit up to which a kernel lets the next one in early: every
kernel sees what the one before it wrote, launched and replayed from a graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2047, 2048, 2049, 8200])
def test_lookup_norm_and_sum(cuda_device, rows):
    from frankentorch_b200.ops import kernels as K
    d = 64
    g = torch.Generator(device=cuda_device).manual_seed(rows)
    wte = torch.randn(300, d, generator=g, device=cuda_device).to(torch.bfloat16)
    wpe = torch.randn(rows, d, generator=g, device=cuda_device).to(torch.bfloat16)
    gamma, beta = (torch.randn(d, generator=g, device=cuda_device).to(torch.bfloat16) for _ in range(2))
    ids = torch.randint(0, 300, (1, rows), generator=g, device=cuda_device)

    def chain():
        x = K.embedding_fwd(ids, wte, wpe, rows)
        y = K.layernorm_fwd(x, gamma, beta)[0]
        return x, y, K.colsum(K.add(y, x))

    first = chain()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = chain()
    for _ in range(3):
        for t in held:
            t.zero_()
        graph.replay()
        for a, b in zip(held, first):
            assert torch.equal(a, b)
    x, y, total = first
    ref = (wte[ids[0]].double() + wpe.double()).to(torch.bfloat16)
    assert torch.equal(x, ref)
    ref_y = torch.nn.functional.layer_norm(x.double(), (d,), gamma.double(), beta.double(), 1e-5)
    assert float((y.double() - ref_y).norm()) <= 2.0 ** -8 * float(ref_y.norm())          # one rounding to bf16
    ref_sum = (y.double() + x.double()).to(torch.bfloat16).double().sum(0)
    assert float((total.double() - ref_sum).norm()) <= 1e-5 * float(ref_sum.norm()) + 1e-3
    K.check_status()
