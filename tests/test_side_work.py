"""Order and lifetime of the weight gradients that run beside the backward pass, on streams that only keep the books: each
knows which launches it is ordered behind, so a missing wait shows as a launch that is not among them."""

import contextlib

import pytest
import torch

from speculators_b200 import ops


class _Stream:
    device, device_index = torch.device("cpu"), 0

    def __init__(self, *_):
        self.cuda_stream, self.behind = id(self), set()

    def wait_stream(self, other):
        self.behind |= other.behind

    def record_event(self):
        event = _Stream()
        event.behind |= self.behind
        return event

    wait_event = wait_stream


@pytest.fixture
def streams(monkeypatch):
    """``caller`` (where ``backward()`` is called) and ``main`` (where forward ran, and so the backward nodes)."""
    caller, main, now = _Stream(), _Stream(), []
    now.append(caller)

    @contextlib.contextmanager
    def stream(s):
        now.append(s)
        yield
        now.pop()

    monkeypatch.setattr(torch.cuda, "Stream", _Stream)
    monkeypatch.setattr(torch.cuda, "stream", stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *_: now[-1])
    monkeypatch.setattr(ops, "_SIDE_STREAMS", {})
    return caller, main


def _weight(width=64):
    """2048 wide its uses are gathered, 64 wide each is launched when it comes."""
    w = torch.nn.Parameter(torch.ones(1, 1).expand(width, width))
    w._flat_grad, w._grad_fresh = torch.zeros(1, 1).expand(width, width), True
    return w


class _Use(torch.autograd.Function):
    """A product with ``weight`` whose gradient is noted as a launch called ``name`` on the stream that it runs on."""

    @staticmethod
    def forward(ctx, x, weight, main, name, then):
        ctx.args = weight, main, name, then
        return x.clone()

    @staticmethod
    def backward(ctx, d):
        weight, main, name, then = ctx.args
        with torch.cuda.stream(main):
            ops._gather_use(weight, (None, None), (d.clone(), d.clone()), lambda uses: torch.cuda.current_stream().behind.add(name))
            if then is not None:
                then(d)
        return d, None, None, None, None


def _use(x, weight, main, name, then=None):
    ops._note_use(weight, None, None)
    return _Use.apply(x, weight, main, name, then)


@pytest.mark.parametrize("width", [64, 2048])
def test_the_stream_that_called_backward_waits_for_the_gradients(streams, width):
    caller, main = streams
    w, x = _weight(width), torch.ones(4, 64, requires_grad=True)
    ops._note_use(w, None, None)  # a use that no gradient comes back from: what is gathered waits for it to the end of the pass
    caller.behind.add("accumulated")  # what autograd has put into the buffer itself on the stream that called it
    behind = []
    _use(x, w, main, "dw", then=lambda _: behind.append("dw" in ops._SIDE_STREAMS[0, main.cuda_stream].behind)).sum().backward()
    assert behind == [width == 64]
    assert "dw" in main.behind and "dw" in caller.behind
    assert width == 64 or "accumulated" in ops._SIDE_STREAMS[0, main.cuda_stream].behind


@pytest.mark.parametrize("rows", [(None, None), (0, 32)])
def test_a_gradient_on_the_main_stream_comes_behind_those_beside_it(streams, rows):
    """A use whose operands the kernel does not take (the library product) after one that it does."""
    _, main = streams
    w, x = _weight(), torch.ones(4, 64, requires_grad=True)
    w._flat_grad = torch.zeros(64, 64)
    before = []

    def library(d):
        r0, r1 = rows
        ops._linear_backward(x.detach(), w, rows, d if r0 is None else d[:, r0:r1], False, True)
        before.append("dw" in main.behind)

    _use(x, w, main, "dw", library).sum().backward()
    assert before == [True]
