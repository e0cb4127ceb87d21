"""Order and lifetime of the weight gradients that run beside the backward pass, on streams that only keep the books: each
knows which launches it is ordered behind, so a missing wait shows as a launch that is not among them."""

import contextlib
import gc
import weakref

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
    caller, main = _Stream(), _Stream()
    now = [caller]

    @contextlib.contextmanager
    def stream(s):
        now.append(s)
        try:
            yield
        finally:
            now.pop()

    monkeypatch.setattr(torch.cuda, "Stream", _Stream)
    monkeypatch.setattr(torch.cuda, "stream", stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *_: now[-1])
    monkeypatch.setattr(ops, "_SIDE_STREAMS", {})
    monkeypatch.setattr(_Product, "alive", [])
    return caller, main


def _weight(width=64):
    """2048 wide its uses are gathered, 64 wide each is launched when it comes."""
    w = torch.nn.Parameter(torch.ones(1, 1).expand(width, width))
    w._flat_grad, w._grad_fresh = torch.zeros(1, 1).expand(width, width), True
    return w


class _Product(torch.autograd.Function):
    """A use of ``weight`` whose gradient is a launch called ``name`` on the stream that it runs on; ``then`` is called behind it."""

    @staticmethod
    def forward(ctx, x, weight, main, name, then, use):
        ctx.args = weight, main, name, then, use
        return x.clone()

    @staticmethod
    def backward(ctx, d):
        weight, main, name, then, use = ctx.args
        with torch.cuda.stream(main):
            operand = d.clone()
            _Product.alive.append(weakref.ref(operand))
            ops._gather_use(weight, (None, None), use, (operand, operand), lambda uses: torch.cuda.current_stream().behind.add(name))
            del operand
            if then is not None:
                then(d)
        return d, None, None, None, None, None

    alive: list = []


def _product(x, weight, main, name, then=None):
    return _Product.apply(x, weight, main, name, then, ops._note_use(weight, None, None))


def _operands():
    return sum(r() is not None for r in _Product.alive)


@pytest.mark.parametrize("width", [64, 2048])
def test_the_stream_that_called_backward_waits_for_the_gradients(streams, width):
    caller, main = streams
    w, x = _weight(width), torch.ones(4, 64, requires_grad=True)
    unused = ops._note_use(w, None, None)  # no gradient comes back from it: what is gathered waits for it to the end of the pass
    caller.behind.add("accumulated")  # what autograd has put into the buffer itself on the stream that called it
    behind = []
    _product(x, w, main, "dw", then=lambda _: behind.append("dw" in ops._SIDE_STREAMS[0, main.cuda_stream].behind)).sum().backward()
    assert behind == [width == 64] and unused is not None
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
        ops._linear_backward(x.detach(), w, rows, None, d if r0 is None else d[:, r0:r1], False, True)
        before.append("dw" in main.behind)

    _product(x, w, main, "dw", library).sum().backward()
    assert before == [True]


@pytest.mark.parametrize("width", [64, 2048])
def test_operands_are_given_back_while_the_pass_runs(streams, width):
    """Forty layers do not keep forty layers' operands, whether launched at once or gathered, and the main stream is behind the
    launch that read what is given back."""
    _, main = streams
    x = torch.ones(4, 64, requires_grad=True)
    most = []

    def count(_):
        most.append(_operands())
        gone = [f"dw{i}" for i, r in zip(range(39, -1, -1), _Product.alive) if r() is None]
        assert main.behind.issuperset(gone)

    y, weights = x, [_weight(width) for _ in range(40)]
    unused = [ops._note_use(w, None, None) for w in weights]
    for i, w in enumerate(weights):
        y = _product(y, w, main, f"dw{i}", count)
    y.sum().backward()
    assert max(most) <= ops._SIDE_HELD + ops._SIDE_PENDING + 1 and len(unused) == 40
    assert _operands() == 0 and main.behind.issuperset(f"dw{i}" for i in range(40))


@pytest.mark.parametrize("width", [64, 2048])
def test_a_pass_that_an_exception_ends_gives_its_operands_back(streams, width):
    _, main = streams
    w, v, x = _weight(width), _weight(64), torch.ones(4, 64, requires_grad=True)

    def stop(_):
        raise ValueError("stop")

    unused = ops._note_use(w, None, None)
    with pytest.raises(ValueError, match="stop"):
        _product(_product(_product(x, w, main, "a", stop), v, main, "b"), w, main, "c").sum().backward()
    gc.collect()  # the exception's traceback
    assert _operands() == 0 and "b" in main.behind and unused is not None
    # later gradients of the weight are ordered behind what that pass launched, and the next pass does not wait for its uses
    other = _Stream()
    with torch.cuda.stream(other):
        ops._wait_for_side_work(v)
    assert "b" in other.behind
    del unused
    launched = []
    _product(x, w, main, "d", lambda _: launched.append("d" in ops._SIDE_STREAMS[0, main.cuda_stream].behind)).sum().backward()
    assert launched == [True]


def test_a_gradient_outside_a_pass_comes_behind_one_that_an_exception_ended(streams):
    caller, main = streams
    w, x = _weight(), torch.ones(4, 64, requires_grad=True)

    def stop(_):
        raise ValueError("stop")

    with pytest.raises(ValueError, match="stop"):
        _product(x, w, main, "a", stop).sum().backward()
    before = []
    ops._gather_use(w, (None, None), None, (x, x), lambda uses: before.append("a" in caller.behind))
    assert before == [True]
