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
