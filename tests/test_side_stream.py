"""The second stream beside a rule's GEMMs: what it is ordered behind, what is kept for it, and that it changes no bit."""
import threading
from types import SimpleNamespace

import pytest
import torch

from frankentorch_b200.autograd.tape import TensorTape
from frankentorch_b200.ops import _lib, fused
from frankentorch_b200.ops import kernels as K

MAIN, SIDE = 3, 9


class _Library:
    """Stands in for the kernel library: records allocations, launches and the order of the streams as they happen."""

    def __init__(self, fail=False):
        self.events, self.fail = [], fail

    def ftk_colsum_blocks(self, rows):
        return 2

    def ftk_stream_order(self, first, then):
        self.events.append(("order", first, then))
        return 0

    def ftk_colsum_bf16(self, x, out, partial, rows, cols, ld, accumulate, stream):
        self.events.append(("sum", stream))
        return -2 if self.fail else 0

    def ftk_gemm_plan(self, desc, bn, splits):
        bn._obj.value, splits._obj.value = 128, 2
        return 0

    def gemm_packed(self, packed, stream):
        d = _lib.FtkGemmDesc.from_buffer_copy(packed)
        self.events.append(("product", stream, d.reduce_stream if d.workspace else None))
        return 0


@pytest.fixture
def fake(monkeypatch):
    lib = _Library()
    new_empty = torch.Tensor.new_empty

    def recording(self, *a, **k):
        lib.events.append(("take",))
        return new_empty(self, *a, **k)

    monkeypatch.setattr(K, "_bf16", lambda t, name: None)
    monkeypatch.setattr(K, "_stream", lambda: MAIN)
    monkeypatch.setattr(K, "_get_device", lambda: 0)
    monkeypatch.setattr(_lib, "load", lambda *a, **k: lib)
    monkeypatch.setattr(torch.Tensor, "new_empty", recording)
    monkeypatch.setattr(fused.SideWork, "enabled", True)
    monkeypatch.setattr(fused.SideWork, "stream_for", classmethod(lambda cls, device: SimpleNamespace(cuda_stream=SIDE)))
    return lib


def _side():
    return fused.SideWork(TensorTape(), torch.device("cuda", 0))


@pytest.mark.parametrize("bound", [True, False])
def test_the_side_stream_waits_behind_the_scratch(fake, bound):
    """A block that is taken from the main stream's pool may have been freed a moment ago, by any thread that launches there: the
    side stream may write it only behind what the main stream held when the block was taken."""
    dy = torch.zeros(16, 8, dtype=torch.bfloat16)
    with _side() as side:
        for _ in range(2):
            side.colsum(dy, out=torch.zeros(8) if bound else None)
    ev = fake.events
    sums = [i for i, e in enumerate(ev) if e[0] == "sum"]
    assert len(sums) == 2 and all(ev[i] == ("sum", SIDE) for i in sums)
    for n, i in enumerate(sums):
        since = ev[sums[n - 1] + 1 if n else 0:i]
        takes = [j for j, e in enumerate(since) if e[0] == "take"]
        assert takes and ("order", MAIN, SIDE) in since[takes[-1]:]
    assert ev[-1] == ("order", SIDE, MAIN)


def test_the_join_comes_before_the_release(fake):
    """Scratch and operands of the side stream are held until the main stream waits for it, also when a launch fails."""
    dy = torch.zeros(16, 8, dtype=torch.bfloat16)
    side = _side()
    with side:
        out = side.colsum(dy)
        held = list(side._held)
        assert any(t is dy for t in held) and any(t is out for t in held)
        assert any(t.numel() == 2 * 8 for t in held)         # the partial sums
    assert not side._held
    fake.fail = True
    with pytest.raises(K.KernelError):
        with _side() as side:
            side.colsum(dy)
    assert fake.events[-1] == ("order", SIDE, MAIN)


def test_split_reductions_are_joined_and_nothing_else_is(fake):
    """A product whose reduction runs on the side stream is joined; a rule that leaves the side stream alone is neither forked nor joined."""
    dy, x = torch.zeros(2048, 16, dtype=torch.bfloat16), torch.zeros(2048, 24, dtype=torch.bfloat16)
    with _side() as side:
        side.wgrad(dy, x)
    assert [e for e in fake.events if e[0] != "take"] == [("product", MAIN, SIDE), ("order", SIDE, MAIN)]
    fake.events.clear()
    with _side() as side:
        side.wgrad(dy[:64], x[:64])
    assert [e for e in fake.events if e[0] != "take"] == [("product", MAIN, None)]


def test_kernels_of_another_device_keep_to_one_stream(fake, monkeypatch):
    """Tensors of a device that is not the current one: the kernels go to the current device's stream, so nothing is moved aside."""
    monkeypatch.setattr(K, "_get_device", lambda: 1)
    with _side() as side:
        assert not side.on
        side.colsum(torch.zeros(16, 8, dtype=torch.bfloat16))
    assert [e for e in fake.events if e[0] != "take"] == [("sum", MAIN)]


def test_column_sums_aside_without_a_list(fake, monkeypatch):
    """A caller that keeps nothing: the memory of operand, scratch and result is held back until the other stream is done with it."""
    recorded = []
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda handle, device=None: handle)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: recorded.append((t.numel(), s)), raising=False)
    dy = torch.zeros(16, 8, dtype=torch.bfloat16)
    out = K.colsum(dy, stream=SIDE)
    assert sorted(recorded) == [(out.numel(), SIDE), (2 * 8, SIDE), (dy.numel(), SIDE)]
    K.colsum(dy)
    K.colsum(dy, stream=SIDE, keep=[])
    assert len(recorded) == 3


# ------------------------------------------------------------------------------------------------ the rules on a GPU
NAMES = ("x", "w0", "b0", "w1", "b1", "w2", "b2")


def _inputs(device, rows, d, seed):
    g = torch.Generator(device=device).manual_seed(seed)
    shapes = ((rows, d), (d, d), (d,), (4 * d, d), (4 * d,), (d, 4 * d), (d,))
    return [(torch.randn(*s, generator=g, device=device) * s[-1] ** -0.5).to(torch.bfloat16) for s in shapes], \
        (torch.randn(rows, d, generator=g, device=device) * 0.01).to(torch.bfloat16)


def _step(values, gy, bound, queue):
    """A linear layer and an MLP, forward and backward: the outputs and every gradient."""
    tape = TensorTape(grad_dtype=None)
    ids, bufs = [], []
    for name, t in zip(NAMES, values):
        ids.append(tape.leaf(t, requires_grad=True, name=name))
        if bound and name != "x":
            bufs.append(torch.full(t.shape, float("nan"), device=t.device))
            tape.bind_grad_buffer(ids[-1], bufs[-1])
    if queue:
        assert fused.enable_grouped_wgrad(tape)
        tape.wgrad_queue.FLUSH_TILES = 1       # every weight gradient is launched, and its operands dropped, inside its rule
    x, w0, b0, w1, b1, w2, b2 = ids
    y0 = fused.linear(tape, x, w0, b0)
    y = fused.mlp_up_down(tape, y0, w1, b1, w2, b2, y0)
    rep = tape.backward(y, seed=gy)
    grads = [rep.gradient(x)] + (bufs if bound else [rep.gradient(i) for i in ids[1:]])
    return [tape.value(y)] + grads


@pytest.mark.gpu
@pytest.mark.parametrize("rows,d", [(2048, 256), (300, 136), (40, 64)])
@pytest.mark.parametrize("bound,queue", [(True, False), (True, True), (False, False)])
def test_the_side_stream_changes_no_bit(cuda_device, monkeypatch, rows, d, bound, queue):
    values, gy = _inputs(cuda_device, rows, d, 3)
    monkeypatch.setattr(fused.SideWork, "enabled", False)
    refs = _step(values, gy, bound, queue)
    monkeypatch.setattr(fused.SideWork, "enabled", True)
    for _ in range(40):
        got = _step(values, gy, bound, queue)
        assert all(torch.equal(a, b) for a, b in zip(got, refs))
    K.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("bound", [True, False])
def test_two_threads_on_one_stream(cuda_device, monkeypatch, bound):
    """Two threads, each with a tape of its own, on the default stream, where one's freed blocks are the other's scratch."""
    work = [_inputs(cuda_device, rows, 256, 7 + rows) for rows in (2048, 1100)]
    monkeypatch.setattr(fused.SideWork, "enabled", False)
    refs = [_step(*w, bound, False) for w in work]
    monkeypatch.setattr(fused.SideWork, "enabled", True)
    torch.cuda.synchronize()
    bad, errors = [0, 0], []

    def run(i):
        try:
            with torch.cuda.device(cuda_device):
                torch.zeros(1, device=cuda_device)      # the thread's context
                for _ in range(60):
                    got = _step(*work[i], bound, False)
                    bad[i] += not all(torch.equal(a, b) for a, b in zip(got, refs[i]))
        except Exception as e:      # noqa: BLE001
            errors.append(e)
    ts = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    K.check_status()
    assert not errors and bad == [0, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("kept", [True, False])
def test_column_sums_on_another_stream(cuda_device, kept):
    side = torch.cuda.Stream(cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(11)
    for rows, cols in ((4096, 3072), (300, 136), (1, 8)):
        x = torch.randn(rows, cols, generator=g, device=cuda_device).to(torch.bfloat16)
        ref = K.colsum(x)
        for _ in range(20):
            keep = [] if kept else None
            got = K.colsum(x.clone(), stream=side.cuda_stream, keep=keep)
            junk = [torch.full((n,), 7.0, device=cuda_device) for n in (cols, 2 * cols, 64 * cols, rows * cols // 2 + 1)]
            torch.cuda.current_stream().wait_stream(side)
            assert torch.equal(got, ref)
            del keep, junk
    K.check_status()
