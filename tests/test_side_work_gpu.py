"""Weight gradients beside the backward pass, on the GPU: their order against streams that other work runs on."""

import pytest
import torch

from speculators_b200 import ops

pytestmark = pytest.mark.gpu


def _weight(rows, cols):
    w = (torch.randn(rows, cols, device="cuda") * 0.05).bfloat16().requires_grad_()
    w._flat_grad, w._grad_fresh = torch.full_like(w, float("nan")), True
    return w


@pytest.fixture
def late(monkeypatch):
    """Every launch beside the pass starts some ten milliseconds late, so that whoever does not wait reads what was there before."""
    run = ops._SideWork.run

    def slow(self, key):
        with torch.cuda.stream(self.stream):
            torch.cuda._sleep(20_000_000)
        run(self, key)

    monkeypatch.setattr(ops._SideWork, "run", slow)


@pytest.mark.parametrize("rows,cols", [(512, 256), (2048, 2048)])  # launched at once, gathered over the uses
def test_forward_on_one_stream_and_backward_from_another(late, rows, cols):
    torch.manual_seed(rows)
    w = _weight(rows, cols)
    x = torch.randn(300, cols, device="cuda").bfloat16()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        losses = [ops.linear(x, w).float().pow(2).mean() for _ in range(2)]
        loss = losses[0] + losses[1]
    torch.cuda.current_stream().wait_stream(stream)
    loss.backward()
    got = w._flat_grad.float()
    wf = w.detach().float().requires_grad_()
    (2 * (x.float() @ wf.t()).pow(2).mean()).backward()
    # dy is rounded to bf16 and so is the sum: two roundings of 2^-9 of the largest terms, and cancellation in between
    assert (got - wf.grad).abs().max() <= 0.02 * wf.grad.abs().max()


@pytest.mark.parametrize("width,rows", [(1024, 2048), (2048, 512)])  # launched at once, gathered where another use is expected
def test_memory_of_a_pass_does_not_grow_with_its_layers(width, rows):
    """Behind the bounds every further layer adds what its forward pass keeps, and no operands of weight gradients."""
    torch.manual_seed(0)
    x = torch.randn(rows, width, device="cuda").bfloat16()

    def extra(layers):
        weights = [_weight(width, width) for _ in range(layers)]
        ops.linear(x, weights[0]).sum().backward()  # allocations of the first call
        y = x
        for w in weights:
            y = ops.linear(y, w)
        loss = y.sum()
        del y
        torch.cuda.synchronize()
        start = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        loss.backward()
        torch.cuda.synchronize()
        return (torch.cuda.max_memory_allocated() - start) / (rows * width * 2)

    bound = ops._SIDE_HELD + ops._SIDE_PENDING
    # in units of one activation: the pass frees a layer's input for each gradient that it forms
    assert extra(3 * bound) <= extra(bound) + 1


def test_memory_after_a_pass_that_an_exception_ended():
    torch.manual_seed(0)
    w = _weight(512, 512)

    def stop(g):
        raise RuntimeError("stop")

    def failing():
        x = torch.randn(4096, 512, device="cuda").bfloat16().requires_grad_()
        y = ops.linear(x, w)
        y.register_hook(stop)
        with pytest.raises(RuntimeError, match="stop"):
            ops.linear(y, w).sum().backward()

    failing()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for _ in range(3):
        failing()
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == before
    w._grad_fresh = True
    x = torch.randn(64, 512, device="cuda").bfloat16()
    ops.linear(x, w).sum().backward()
    want = torch.ones(64, 512, device="cuda").t() @ x.float()
    assert (w._flat_grad.float() - want).abs().max() <= 0.01 * want.abs().max()


def test_an_exception_inside_a_capture_leaves_the_streams_usable():
    torch.manual_seed(0)
    w = _weight(512, 512)
    x = torch.randn(256, 512, device="cuda").bfloat16().requires_grad_()
    stream = torch.cuda.Stream()

    def step(fail):
        w._grad_fresh = True
        y = ops.linear(x, w)
        if fail:
            y.register_hook(lambda g: (_ for _ in ()).throw(RuntimeError("stop")))
        torch.autograd.backward(ops.linear(y, w).float().pow(2).mean(), inputs=[x, w])

    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step(False)
    torch.cuda.current_stream().wait_stream(stream)
    want = w._flat_grad.clone()
    with pytest.raises(RuntimeError, match="stop"):
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream):
            step(True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        step(False)
    w._flat_grad.fill_(float("nan"))
    graph.replay()
    assert torch.equal(w._flat_grad, want)
    w._flat_grad.fill_(float("nan"))
    step(False)
    assert torch.equal(w._flat_grad, want)
