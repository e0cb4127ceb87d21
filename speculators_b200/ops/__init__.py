"""Hot operators of the framework.

Every function here has two implementations behind one signature:

* CUDA tensors run the hand-written sm_100a kernels of ``csrc/`` through
  ``torch.ops.sb200`` (bf16 storage, fp32 math).  There is no fallback on a GPU:
  a missing extension is a hard error.
* CPU tensors (any float dtype) run a plain PyTorch formulation.  That path is the
  numerical oracle the kernel tests compare against, and it is what the gloo /
  world_size > 1 plumbing tests execute.

All functions are differentiable; the CUDA paths carry their own backward
kernels via ``torch.autograd.Function``.
"""

from __future__ import annotations

import collections
import contextlib
import math
import weakref
from typing import NamedTuple

import torch
import torch.nn.functional as F

from speculators_b200.ops import _ext
from speculators_b200.ops.attention import AttnSpec, masked_attention, masked_attention_reference

__all__ = [
    "AttnSpec",
    "StepRows",
    "LOSS_OPS",
    "adamw_step_",
    "eagle3_input_concat",
    "embedding",
    "fused_row_loss",
    "gated",
    "check_gemm_status",
    "clear_fresh_grad",
    "gemm_status",
    "GroupPlan",
    "grouped_linear",
    "grouped_linear_ok",
    "linear",
    "linear_swiglu",
    "lm_head_loss_ok",
    "lm_head_loss_raw",
    "masked_attention",
    "matmul_nn",
    "matmul_nt",
    "matmul_tn",
    "masked_attention_reference",
    "native",
    "only_live",
    "norm_rope_heads",
    "repeat_rows",
    "rms_norm",
    "rms_norm_fork",
    "rms_norm_pair",
    "rms_norm_taken",
    "rope_",
    "rope_split",
    "split_gated_query",
    "step_rows",
    "sum_of_squares",
    "swiglu",
    "take_rows",
    "token_cross_entropy",
    "ttt_step_loss",
    "ttt_step_tail",
]

LOSS_OPS = {"kl_div": 0, "rkl": 1, "jsd": 2, "ce": 3, "tv": 4}


def native():
    """``torch.ops.sb200`` (builds / loads the extension on first use)."""
    return _ext.lib()


def _use_native(t: torch.Tensor) -> bool:
    return t.is_cuda


# --------------------------------------------------------------------------- linear
_GEMM_STATUS: dict[int, torch.Tensor] = {}


def own_gemm_enabled() -> bool:
    import os

    return os.environ.get("SB200_LINEAR_GEMM", "tcgen05") != "cublas"


def _gemm_operand_ok(t: torch.Tensor) -> bool:
    return (t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0
            and t.data_ptr() % 16 == 0)


def gemm_status(device: torch.device) -> torch.Tensor:
    """The device word the tcgen05 GEMM writes a non-zero code to if one of its bounded
    waits ever runs out (it should stay 0; read it where a host sync is acceptable)."""
    idx = device.index if device.index is not None else torch.cuda.current_device()
    if idx not in _GEMM_STATUS:
        _GEMM_STATUS[idx] = torch.zeros(1, dtype=torch.int32, device=torch.device("cuda", idx))
    return _GEMM_STATUS[idx]


_WAIT_CODES = {
    1: "GEMM producer", 2: "GEMM MMA issuer", 3: "GEMM epilogue", 4: "GEMM partial sums of a divided tile",
    31: "attention forward producer", 32: "attention forward MMA issuer", 33: "attention forward softmax",
    41: "attention dQ producer", 42: "attention dQ MMA issuer", 43: "attention dQ element-wise warps",
    44: "attention dK/dV producer", 45: "attention dK/dV MMA issuer", 46: "attention dK/dV element-wise warps",
    51: "attention (head dim 256) producer", 52: "attention (head dim 256) MMA issuer", 53: "attention (head dim 256) element-wise warps",
}


def check_gemm_status() -> None:
    """Raise if a tcgen05 kernel (GEMM or attention) launched by this process reported a wait
    that ran out; the kernels share one status word per device."""
    for idx, word in _GEMM_STATUS.items():
        code = int(word.item())
        if code:
            word.zero_()
            raise RuntimeError(f"a tcgen05 kernel on cuda:{idx} gave up waiting (code {code}: {_WAIT_CODES.get(code, 'unknown wait')})")


# ``live`` (here and below): an int32 tensor on the device that says how many of the rows hold anything (``step_rows``).  The
# kernels neither read nor write the rows behind; what runs elsewhere takes all rows, and a sum over rows leaves those out.
def only_live(x2: torch.Tensor, live: torch.Tensor | None) -> torch.Tensor:
    """``x2`` (rows first) with zeros in the rows from ``live`` on."""
    if live is None:
        return x2
    used = torch.arange(x2.shape[0], device=x2.device) < live
    return torch.where(used.view(-1, *[1] * (x2.dim() - 1)), x2, torch.zeros((), dtype=x2.dtype, device=x2.device))


def _settled(d: torch.Tensor | None, live: torch.Tensor | None) -> torch.Tensor | None:
    """A gradient that a backward pass hands on.  Nothing reads its rows from ``live`` on but autograd's anomaly detection, which
    looks for NaN in all of them: zeros for it."""
    return d if d is None or live is None or not (torch.is_anomaly_enabled() and torch.is_anomaly_check_nan_enabled()) else only_live(d, live)


def _forward_gemm(x2: torch.Tensor, w: torch.Tensor, residual: torch.Tensor | None, live: torch.Tensor | None = None) -> torch.Tensor:
    """``x2 @ w.T (+ residual)`` for 2-D operands.  bf16 CUDA operands with 16-byte aligned
    rows run on the package's tcgen05 kernel (the residual is read in its epilogue, no
    copy of it is made); everything else goes to the library."""
    if _gemm_operand_ok(x2) and _gemm_operand_ok(w) and own_gemm_enabled() and (
        residual is None or (_gemm_operand_ok(residual) and residual.shape == (x2.shape[0], w.shape[0]))
    ):
        out = torch.empty((x2.shape[0], w.shape[0]), dtype=x2.dtype, device=x2.device)
        native().gemm_tn(x2, w, out, residual, 2 if residual is not None else 0, gemm_status(x2.device), live)
        return out
    if residual is not None:
        return torch.addmm(residual, x2, w.t())
    return x2 @ w.t()


def _dgrad_gemm(dy2: torch.Tensor, w: torch.Tensor, out: torch.Tensor | None = None, accumulate: bool = False,
                live: torch.Tensor | None = None) -> torch.Tensor:
    """``dy2 @ w`` (input gradient of a linear layer) on the tcgen05 kernel: the weight is read
    as stored, ``[out, in]`` with ``in`` contiguous, as an MN-major B operand."""
    dx = out if out is not None else torch.empty((dy2.shape[0], w.shape[1]), dtype=dy2.dtype, device=dy2.device)
    native().gemm(dy2, w, dx, 1 if accumulate else 0, False, True, gemm_status(dy2.device), live)
    return dx


def _wgrad_gemm(dy2: torch.Tensor, x2: torch.Tensor, out: torch.Tensor | None, accumulate: bool, live: torch.Tensor | None = None) -> torch.Tensor:
    """``dy2.T @ x2`` (weight gradient) on the tcgen05 kernel, both operands read in place as
    MN-major tiles, stored into or added to ``out`` in the epilogue."""
    if out is None:
        out = torch.empty((dy2.shape[1], x2.shape[1]), dtype=dy2.dtype, device=dy2.device)
    native().gemm(dy2, x2, out, 1 if accumulate else 0, True, True, gemm_status(dy2.device), live)
    return out


def matmul_nt(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """``a @ b.T`` for 2-D tensors; bf16 CUDA operands with aligned rows use the tcgen05 kernel."""
    if _gemm_operand_ok(a) and _gemm_operand_ok(b) and own_gemm_enabled():
        return _forward_gemm(a, b, None)
    return a @ b.t()


def matmul_nn(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor | None = None, accumulate: bool = False) -> torch.Tensor:
    """``a @ b`` for 2-D tensors (``b`` read as stored, no transpose copy), optionally stored
    into / added to ``out``."""
    if _gemm_operand_ok(a) and _gemm_operand_ok(b) and own_gemm_enabled() and (out is None or _gemm_operand_ok(out)):
        return _dgrad_gemm(a, b, out, accumulate)
    if out is None:
        return a @ b
    return out.addmm_(a, b) if accumulate else torch.mm(a, b, out=out)


def matmul_tn(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor | None = None, accumulate: bool = False) -> torch.Tensor:
    """``a.T @ b`` for 2-D tensors, optionally stored into / added to ``out``."""
    if _gemm_operand_ok(a) and _gemm_operand_ok(b) and own_gemm_enabled() and (out is None or _gemm_operand_ok(out)):
        return _wgrad_gemm(a, b, out, accumulate)
    if out is None:
        return a.t() @ b
    return out.addmm_(a.t(), b) if accumulate else torch.mm(a.t(), b, out=out)


# --------------------------------------------------------------------------- grouped (expert) linears
class GroupPlan:
    """Padded row order of a grouped product, all on the device: expert ``e`` owns the rows
    ``seg[e] .. seg[e] + counts[e]`` of a ``[capacity, .]`` buffer, ``seg[e]`` a multiple of 128,
    the rows up to ``seg[e + 1]`` are zero.  ``dest[i]`` is the padded row of the ``i``-th row of
    the expert-sorted order.  Built without reading anything back to the host."""

    def __init__(self, counts: torch.Tensor, num_rows: int):
        counts32 = counts.to(torch.int32).contiguous()
        E = counts32.numel()
        self.seg, self.mtile_start = native().moe_group_plan(counts32)
        self.capacity = (num_rows + 127 * E + 127) // 128 * 128  # worst case: every expert's tail padded by 127 rows
        start = torch.cumsum(counts32, 0) - counts32  # unpadded offsets
        expert_of = torch.repeat_interleave(torch.arange(E, device=counts.device), counts32.long(), output_size=num_rows)
        self.dest = (torch.arange(num_rows, device=counts.device) - start[expert_of] + self.seg[expert_of]).long()

    def pad(self, x_sorted: torch.Tensor) -> torch.Tensor:
        out = x_sorted.new_zeros((self.capacity, x_sorted.shape[1]))
        return out.index_copy(0, self.dest, x_sorted)

    def unpad(self, y_padded: torch.Tensor) -> torch.Tensor:
        return _UnpadRowsFn.apply(y_padded, self.dest)


class _UnpadRowsFn(torch.autograd.Function):
    """``y_padded[dest]`` for distinct ``dest``: the gradient is a row copy into zeros, where autograd's
    ``index_select`` backward would add with atomics (0.67 ms against 0.23 ms for 40960 x 2048 rows)."""

    @staticmethod
    def forward(ctx, y_padded, dest):
        ctx.save_for_backward(dest)
        ctx.rows = y_padded.shape[0]
        return y_padded.index_select(0, dest)

    @staticmethod
    def backward(ctx, dy):
        (dest,) = ctx.saved_tensors
        return dy.new_zeros((ctx.rows, dy.shape[1])).index_copy_(0, dest, dy), None


class _GroupedLinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x_pad, weight, seg, mts):
        out = torch.empty((x_pad.shape[0], weight.shape[1]), dtype=x_pad.dtype, device=x_pad.device)
        native().gemm_grouped_rows(x_pad, weight, out, False, seg, mts, gemm_status(x_pad.device))
        ctx.save_for_backward(x_pad, weight, seg, mts)
        return out

    @staticmethod
    def backward(ctx, dy):
        x_pad, weight, seg, mts = ctx.saved_tensors
        dy = dy if (dy.stride(-1) == 1 and dy.stride(0) % 8 == 0 and dy.data_ptr() % 16 == 0) else dy.contiguous()
        status = gemm_status(dy.device)
        dx = dw = None
        if ctx.needs_input_grad[0]:
            dx = torch.empty_like(x_pad)
            native().gemm_grouped_rows(dy, weight, dx, True, seg, mts, status)
        if ctx.needs_input_grad[1]:
            dw, accumulate, attached = _param_grad_target(weight)
            native().gemm_grouped_wgrad(dy, x_pad, dw, accumulate, seg, mts, status)
            dw = None if attached else dw
        return dx, dw, None, None


def grouped_linear_ok(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether ``grouped_linear`` can run on the tcgen05 kernel for these operands."""
    return (own_gemm_enabled() and _gemm_operand_ok(x) and weight.is_cuda and weight.dtype == torch.bfloat16 and weight.dim() == 3
            and weight.is_contiguous() and weight.shape[1] % 256 == 0 and weight.shape[2] % 256 == 0 and x.shape[0] % 128 == 0)


def grouped_linear(x_pad: torch.Tensor, weight: torch.Tensor, plan: GroupPlan) -> torch.Tensor:
    """``y[r] = weight[e(r)] @ x_pad[r]`` for rows in the padded expert order of ``plan``
    (``weight``: ``[E, out, in]``).  Forward, input gradient and per-expert weight gradient are
    grouped launches of the tcgen05 GEMM whose tile schedule reads the experts' row counts from
    device memory, so the call has fixed shapes and no host synchronisation."""
    return _GroupedLinearFn.apply(x_pad, weight, plan.seg, plan.mtile_start)


class _LinearFn(torch.autograd.Function):
    """``y = x @ W[rows].T (+ residual)`` with the weight gradient accumulated in place.

    When the training engine has attached a flat gradient view to the weight
    (``weight._flat_grad``), backward runs ``grad[rows].addmm_(dy.T, x)``: one GEMM
    whose epilogue adds into the gradient buffer, instead of a GEMM into a temporary
    followed by autograd's separate accumulation pass over the whole weight.  The
    residual, when given, rides in the forward GEMM's epilogue (``beta = 1``).
    """

    @staticmethod
    def forward(ctx, x, weight, residual, r0, r1, use, live):
        # x is [rows, in]; the result is a fresh tensor (never a view), so callers may
        # rotate / normalise it in place
        w = weight if r0 is None else weight[r0:r1]
        y = _forward_gemm(x, w, residual, live)
        ctx.save_for_backward(x, weight, live)
        ctx.rows, ctx.use = (r0, r1), use
        ctx.has_residual = residual is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        x2, weight, live = ctx.saved_tensors
        dx, dw = _linear_backward(x2, weight, ctx.rows, ctx.use, dy, ctx.needs_input_grad[0], ctx.needs_input_grad[1], live)
        dres = dy if ctx.has_residual and ctx.needs_input_grad[2] else None
        return dx, dw, dres, None, None, None, None


_MAX_USES = 4  # of a weight in one product (the kernel's operand maps)
# Half a wave of 256 x 256 tiles: below, the product runs on smaller tiles use by use, and is best started at once
_GATHER_ELEMENTS = 37 * 65536


class _SideWork:
    """Weight gradients of one backward pass: gathered over the uses of a weight, run on a stream of their own.

    The pass's own end-of-pass callback holds the only reference that lasts, so a pass that an exception ends gives its
    operands back when the engine drops it."""

    def __init__(self, main: torch.cuda.Stream, at: tuple[int, int]):
        self.main = main
        self.stream = _SIDE_STREAMS.get(at)
        if self.stream is None:
            self.stream = _SIDE_STREAMS[at] = torch.cuda.Stream(main.device)
        self.held: collections.deque = collections.deque()  # (event behind a launch, its operands, itself with what it reads), the oldest first
        self.weights: list[torch.Tensor] = []
        self.pending: dict[tuple, tuple] = {}  # (weight's id, rows) -> (weight, uses gathered, launch)

    def run(self, key: tuple) -> None:
        weight, uses, launch = self.pending.pop(key)
        self.stream.wait_stream(self.main)
        with torch.cuda.stream(self.stream):
            _wait_for_side_work(weight)  # of another stream's pass
            launch(uses)
        self.weights.append(weight)
        weight._side_stream = self.stream
        self.held.append((self.stream.record_event(), uses, launch))
        while len(self.held) > _SIDE_HELD:
            self.main.wait_event(self.held[0][0])  # the memory goes back to the main stream's order
            self.held.popleft()

    def finish(self) -> None:
        # The engine runs this on the stream that ``backward()`` was called on, once that stream waits for those of the leaves.
        # It is not ``main`` where forward ran on another one, and whoever reads the gradients reads them there.
        current = torch.cuda.current_stream(self.main.device)
        if self.pending and current != self.main:
            self.stream.wait_stream(current)  # gradients of the same weights that came through autograd's own accumulation
        for key in list(self.pending):
            self.run(key)
        self.main.wait_stream(self.stream)
        if current != self.main:
            current.wait_stream(self.main)
        for w in self.weights:
            if w._side_stream is self.stream:
                w._side_stream = None
        self.held.clear()

    def __del__(self):
        if self.held:  # the pass did not come to its end
            with contextlib.suppress(RuntimeError):  # a capture that the exception ended, too
                self.main.wait_stream(self.stream)


_SIDE_STREAMS: dict[tuple[int, int], torch.cuda.Stream] = {}  # by device and main stream (torch hands out streams from a fixed pool)
# by device, main stream and backward pass (threads may run several at once)
_SIDE_WORK: weakref.WeakValueDictionary[tuple[int, int, int], _SideWork] = weakref.WeakValueDictionary()
# Bounds on what a pass keeps allocated for its weight gradients, however deep the model: operands of launches that the main
# stream has not waited for yet, and weights with uses gathered but not launched.  Four launches are a layer's.  Bounds of 1 to 8
# take the same time, and most steps the same as without one (70B-shaped layer 33.3 ms); five layers of 8192 rows are 2 % faster
# with one (57.4 ms, 58.6 without), and the smallest step's chain feels a wait for every launch (0.441 ms, 0.445 at a bound of 1).
_SIDE_HELD = 4
_SIDE_PENDING = 16


def _wait_for_side_work(weight: torch.Tensor) -> None:
    stream = getattr(weight, "_side_stream", None)
    if stream is not None:
        current = torch.cuda.current_stream(weight.device)
        if current != stream:
            current.wait_stream(stream)


class _Use:
    """A differentiated product's use of a weight (or of rows of it) whose gradient is still to come: held by the product's
    node, so that it goes with the graph if no gradient comes."""

    def __init__(self, weight: torch.Tensor, rows: tuple):
        self.counts, self.rows = weight.__dict__.setdefault("_grad_uses", {}), rows
        self.counts[rows] = self.counts.get(rows, 0) + 1

    def left(self) -> int:
        """Count this use as come; how many others of the same rows are still to come."""
        counts, self.counts = self.counts, None
        if counts is None:  # the node's second pass
            return 0
        n = counts[self.rows] - 1
        if n:
            counts[self.rows] = n
        else:
            del counts[self.rows]
        return n

    def __del__(self):
        self.left()


def _note_use(weight: torch.Tensor, *rows) -> _Use | None:
    """Called where a differentiated product uses ``weight`` (or rows of it): for the product's node to keep."""
    return _Use(weight, rows) if getattr(weight, "_flat_grad", None) is not None else None


def _gather_use(weight: torch.Tensor, rows: tuple, use: _Use | None, operands: tuple, launch) -> None:
    """One use's operands of a gradient that goes into the flat buffer.  ``launch(uses)`` forms the gradient of all uses as one
    product once the last expected one (or ``_MAX_USES``) has come: training-time-test passes read and wrote every gradient
    once a pass.  It runs beside the rest of the backward pass, where nothing needs its result: on its own stream it fills
    the SMs that the chain of input gradients leaves idle - the last wave of a product, the short element-wise kernels.
    Waiting for further uses does not pay for small weights (``_GATHER_ELEMENTS``), whose products are bound by neither.  The
    pass's end runs what is left and joins the streams, and so does any other gradient of the same weight."""
    left = use.left() if use is not None else 0
    task = torch._C._current_graph_task_id()
    if task < 0:  # a node's backward called by hand
        _wait_for_side_work(weight)  # of a pass that an exception ended
        launch([operands])
        return
    main = torch.cuda.current_stream(weight.device)
    at = (main.device_index, main.cuda_stream, task)
    work = _SIDE_WORK.get(at)
    if work is None:
        work = _SIDE_WORK[at] = _SideWork(main, at[:2])
        torch.autograd.Variable._execution_engine.queue_callback(work.finish)
    key = (id(weight), *rows)
    _, uses, _ = work.pending.setdefault(key, (weight, [], launch))
    uses.append(operands)
    # Three uses as one product against three, weights of 4096 x 4096 to 57344 x 8192: of 736 rows 1.7 to 2.1 times as fast, of
    # 2048 rows 1.04 to 1.16, of 4096 1.01 to 1.05, of 6144 0.996 to 1.03, of 8192 1.01 to 1.02 (28672 x 4096: 665 and 388 us,
    # 1106 and 1049, 1989 and 1949, 2835 and 2846, 4134 and 4104).  Past 6144 rows that is within the spread of the runs and not
    # worth keeping the uses' operands for; only the smallest that are gathered would still gain there (2048 x 2048, 8192 rows:
    # 1.16, some 25 us).  Rows grouped by expert are few for each.
    whole = weight.numel() < _GATHER_ELEMENTS or (weight.dim() == 2 and operands[0].shape[0] > 6144)
    if left == 0 or len(uses) == _MAX_USES or whole:
        work.run(key)
    elif len(work.pending) > _SIDE_PENDING:
        work.run(next(iter(work.pending)))


def _linear_backward(x2, weight, rows, use, dy, need_dx: bool, need_dw: bool, live=None):
    """``(dx, dw)`` of ``y = x2 @ weight[rows].T``; ``dw`` is ``None`` when the gradient went
    straight into the flat buffer the training engine attached to the weight.  ``use``: what ``_note_use`` gave the product."""
    r0, r1 = rows
    w = weight if r0 is None else weight[r0:r1]
    dy2 = dy if (dy.stride(-1) == 1 and dy.stride(0) % 8 == 0 and dy.data_ptr() % 16 == 0) else dy.contiguous()
    dx = dw = None
    own = own_gemm_enabled() and _gemm_operand_ok(dy2) and _gemm_operand_ok(w) and _gemm_operand_ok(x2)
    if need_dx:
        dx = _dgrad_gemm(dy2, w, live=live) if own else dy2 @ w
    if need_dw and not own:
        dy2, x2 = only_live(dy2, live), only_live(x2, live)
    if need_dw:
        flat = getattr(weight, "_flat_grad", None)
        if flat is not None and own and _gemm_operand_ok(flat if r0 is None else flat[r0:r1]) and x2.shape[0] > 0:
            def launch(uses):
                # the first gradient of these rows since the engine's zero_grad, which left the buffer uncleared, is stored
                target, accumulate = _param_grad_target(weight, beside=True)[:2] if r0 is None else _row_grad_target(weight, r0, r1, beside=True)
                status = gemm_status(target.device)
                all_rows = status[:0]
                native().gemm_wgrad_parts_rows([u[0] for u in uses], [u[1] for u in uses], target, accumulate, status,
                                               [all_rows if u[2] is None else u[2] for u in uses])

            _gather_use(weight, (r0, r1), use, (dy2, x2, live), launch)
        elif flat is not None:
            if use is not None:
                use.left()
            dy2, x2 = (only_live(t, live if own else None) for t in (dy2, x2))
            target, accumulate = _param_grad_target(weight)[:2] if r0 is None else _row_grad_target(weight, r0, r1)
            if accumulate:
                target.addmm_(dy2.t(), x2)
            else:
                torch.mm(dy2.t(), x2, out=target)
        elif r0 is None:
            dw = _wgrad_gemm(dy2, x2, None, accumulate=False, live=live) if own else dy2.t() @ x2
        else:
            dw = torch.zeros_like(weight)
            if own and _gemm_operand_ok(dw[r0:r1]):
                _wgrad_gemm(dy2, x2, dw[r0:r1], accumulate=False, live=live)
            else:
                dy2, x2 = (only_live(t, live if own else None) for t in (dy2, x2))
                dw[r0:r1] = dy2.t() @ x2
    return _settled(dx, live), dw


def linear(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None, residual: torch.Tensor | None = None,
           rows: tuple[int, int] | None = None, live: torch.Tensor | None = None) -> torch.Tensor:
    """``x @ weight[rows].T (+ bias) (+ residual)``.  On CUDA in bf16 the forward product
    runs on the package's tcgen05 GEMM with the residual read in its epilogue
    (``SB200_LINEAR_GEMM=cublas`` sends it to the library instead); the two backward
    products run on the same kernel with the transposed operands read in place (MN-major
    tiles), the weight gradient accumulating in the epilogue into the engine's flat
    gradient buffer.  ``live``: see ``step_rows`` (no bias then)."""
    if live is not None and bias is not None:
        raise ValueError("linear: a bias takes all rows")
    if x.is_cuda and (weight.requires_grad or x.requires_grad) and torch.is_grad_enabled():
        r0, r1 = rows if rows is not None else (None, None)
        lead = x.shape[:-1]
        x2 = x.reshape(-1, x.shape[-1])
        res2 = residual.reshape(-1, residual.shape[-1]) if residual is not None else None
        y = _LinearFn.apply(x2, weight, res2, r0, r1, _note_use(weight, r0, r1) if weight.requires_grad else None, live)
        if len(lead) != 1:
            y = y.view(*lead, y.shape[-1])
        if bias is not None:
            y = y + (bias if rows is None else bias[rows[0] : rows[1]])
        return y
    w = weight if rows is None else weight[rows[0] : rows[1]]
    b = bias if (bias is None or rows is None) else bias[rows[0] : rows[1]]
    if x.is_cuda and x.dtype == torch.bfloat16 and b is None and not torch.is_grad_enabled() and own_gemm_enabled():
        x2 = x.reshape(-1, x.shape[-1])
        res2 = residual.reshape(-1, residual.shape[-1]) if residual is not None else None
        return _forward_gemm(x2, w, res2, live).view(*x.shape[:-1], w.shape[0])
    y = F.linear(x, w, b)
    return y if residual is None else y + residual


# --------------------------------------------------------------------------- rmsnorm
_RMSNORM_MAX_WIDTH = 32768


def _rms_norm_ref(x: torch.Tensor, weight: torch.Tensor, eps: float, centred: bool = False) -> torch.Tensor:
    dt = x.dtype
    xf = x.float()
    xf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)
    return (xf * (1.0 + weight.float())).to(dt) if centred else weight * xf.to(dt)


def _grad_rows(d: torch.Tensor | None, width: int) -> torch.Tensor | None:
    """A gradient as the ``[rows, width]`` layout the kernels read."""
    if d is None:
        return None
    d2 = d.reshape(-1, width)
    return d2 if d2.stride(-1) == 1 and d2.stride(0) % 8 == 0 and d2.data_ptr() % 16 == 0 else d2.contiguous()


def _param_grad_target(weight: torch.Tensor, beside: bool = False) -> tuple[torch.Tensor, bool, bool]:
    """Where a kernel puts a parameter's gradient: ``(buffer, accumulate, attached)``.  With a flat gradient view attached
    by the training engine that view (stored into by the first gradient after ``zero_grad``, which left it uncleared, added
    to by later ones; autograd then gets ``None``), else a fresh tensor.  ``beside``: called by what ``_gather_use`` runs."""
    if not beside:
        _wait_for_side_work(weight)
    flat = getattr(weight, "_flat_grad", None)
    if flat is None:
        return torch.empty_like(weight), False, False
    fresh = getattr(weight, "_grad_fresh", False) is True
    if fresh:
        weight._grad_fresh = False
    else:
        clear_fresh_grad(weight)
    return flat, not fresh, True


def gradient_watched(p: torch.Tensor) -> bool:
    """Whether a hook of the caller's waits for the gradient of ``p`` (the training engine's own does not count): a gradient that
    goes straight into the flat buffer passes it by."""
    hooks = (p._backward_hooks or {}).values()  # noqa: SLF001
    return any(not getattr(h, "of_engine", False) for h in hooks) or bool(getattr(p, "_post_accumulate_grad_hooks", None))


def clear_fresh_grad(p: torch.Tensor) -> None:
    """Zero what no gradient has been stored into since the engine's ``zero_grad``: all of the flat view
    (``_grad_fresh`` is ``True``) or the row intervals that ``_row_grad_target`` has left."""
    _wait_for_side_work(p)
    fresh = getattr(p, "_grad_fresh", False)
    if fresh is False:
        return
    p._grad_fresh = False
    for r0, r1 in [(0, p.shape[0])] if fresh is True else fresh:
        p._flat_grad[r0:r1].zero_()


def _row_grad_target(weight: torch.Tensor, r0: int, r1: int, beside: bool = False) -> tuple[torch.Tensor, bool]:
    """``(rows of the flat gradient view, accumulate)`` for a gradient of rows ``r0 .. r1`` alone: stored where nothing has been
    stored since ``zero_grad``; the intervals still unwritten stay noted on the weight.  ``beside`` as in ``_param_grad_target``:
    anyone else waits for what earlier uses of the rows have launched."""
    if not beside:
        _wait_for_side_work(weight)
    fresh = getattr(weight, "_grad_fresh", False)
    if fresh is True:
        fresh = [(0, weight.shape[0])]
    inside = [iv for iv in fresh or [] if iv[0] <= r0 and r1 <= iv[1]]
    if not inside:
        if any(a < r1 and r0 < b for a, b in fresh or []):  # partly written
            clear_fresh_grad(weight)
        return weight._flat_grad[r0:r1], True
    (a, b), = inside
    rest = [iv for iv in fresh if iv != (a, b)] + [iv for iv in ((a, r0), (r1, b)) if iv[0] < iv[1]]
    weight._grad_fresh = rest or False
    return weight._flat_grad[r0:r1], False


def _norm_backward(dy, dy2, x2, weight, rstd, residual_grad, need_dx: bool, need_dw: bool, centred: bool, live=None):
    """``(dx, dw)`` of a norm over ``x2 [rows, H]``; ``dw`` is ``None`` when it went into the engine's flat buffer."""
    dx = torch.empty_like(x2) if need_dx else None
    dw, accumulate, attached = _param_grad_target(weight) if need_dw else (None, False, False)
    if need_dx or need_dw:
        native().rmsnorm_bwd(dy, dy2, x2, weight, rstd, residual_grad if need_dx else None, dx, dw, accumulate, centred, live)
    return _settled(dx, live), None if attached else dw


class _RMSNormPairFn(torch.autograd.Function):
    """Norm of ``x`` handed out twice, for two consumers whose gradients meet in the backward kernel."""

    @staticmethod
    def forward(ctx, x, weight, eps, live):
        y = torch.empty_like(x)
        rstd = torch.empty(x.shape[0], dtype=torch.float32, device=x.device)
        native().norm_fwd(x, weight, None, y, rstd, eps, False, live)
        ctx.save_for_backward(x, weight, rstd, live)
        ctx.set_materialize_grads(False)
        return y, y.view_as(y)

    @staticmethod
    def backward(ctx, d1, d2):
        d1, d2 = (d1, d2) if d1 is not None else (d2, None)
        if d1 is None:
            return None, None, None, None
        x, weight, rstd, live = ctx.saved_tensors
        H = x.shape[1]
        return *_norm_backward(_grad_rows(d1, H), _grad_rows(d2, H), x, weight, rstd, None, ctx.needs_input_grad[0], ctx.needs_input_grad[1], False, live), None, None


def rms_norm_pair(x: torch.Tensor, weight: torch.Tensor, eps: float, live: torch.Tensor | None = None) -> tuple[torch.Tensor, torch.Tensor]:
    """``rms_norm(x)`` twice, for two consumers."""
    if _norm_native(x) and x.dim() == 2 and x.is_contiguous() and torch.is_grad_enabled() and x.requires_grad:
        return _RMSNormPairFn.apply(x, weight, eps, live)
    y = rms_norm(x, weight, eps, live=live)
    return y, y


class _RMSNormFn(torch.autograd.Function):
    """Norm of ``x``; with ``fork`` the result is ``(normalised, x)`` and the gradient that comes back through the second
    (a residual branch) is added inside the norm's backward kernel instead of a pass of autograd's own."""

    @staticmethod
    def forward(ctx, x, weight, eps, centred, fork, live):
        H = x.shape[-1]
        x2 = x.reshape(-1, H)
        if x2.stride(-1) != 1 or x2.stride(0) % 8 or x2.data_ptr() % 16:
            x2 = x2.contiguous()
        # allocated in the caller's shape and returned as it is: a view made in here could not be
        # modified in place afterwards (the rotary kernel does that to normalised q / k heads)
        y = torch.empty(x.shape, dtype=x.dtype, device=x.device)
        rstd = torch.empty(x2.shape[0], dtype=torch.float32, device=x.device)
        native().norm_fwd(x2, weight, None, y.view(-1, H), rstd, eps, centred, live)
        ctx.save_for_backward(x2, weight, rstd, live)
        ctx.shape, ctx.centred = x.shape, centred
        ctx.set_materialize_grads(False)
        return (y, x.view_as(x)) if fork else y

    @staticmethod
    def backward(ctx, dy, dres=None):
        if dy is None:
            return dres, None, None, None, None, None
        x2, weight, rstd, live = ctx.saved_tensors
        H = x2.shape[-1]
        dx, dw = _norm_backward(_grad_rows(dy, H), None, x2, weight, rstd, _grad_rows(dres, H), ctx.needs_input_grad[0], ctx.needs_input_grad[1], ctx.centred,
                                live)
        return (dx.view(ctx.shape) if dx is not None else None), dw, None, None, None, None


def _norm_native(x: torch.Tensor) -> bool:
    return _use_native(x) and x.dtype == torch.bfloat16 and x.shape[-1] <= _RMSNORM_MAX_WIDTH and x.shape[-1] % 8 == 0


def rms_norm(x: torch.Tensor, weight: torch.Tensor, eps: float, centred: bool = False, live: torch.Tensor | None = None) -> torch.Tensor:
    """RMSNorm over the last dim: ``weight * (x / rms(x))`` with fp32 statistics (``centred``: ``(1 + weight)``, applied
    before rounding).  bf16 CUDA rows of up to 32768 elements run on the package's kernels (one row per CTA with the row in
    registers; one row per warp for rows of up to 256)."""
    if _norm_native(x):
        return _RMSNormFn.apply(x, weight, eps, centred, False, live)
    return _rms_norm_ref(x, weight, eps, centred)


def add_rms_norm(x: torch.Tensor, add: torch.Tensor, weight: torch.Tensor, eps: float) -> tuple[torch.Tensor, torch.Tensor]:
    """``(x + add, rms_norm(x + add))``, in one launch where no gradient is asked for."""
    if (_norm_native(x) and not torch.is_grad_enabled() and x.dim() == 2 and x.shape[1] > 256 and add.shape == x.shape and add.dtype == x.dtype
            and weight.dtype == x.dtype and all(t.device == x.device and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in (x, add, weight))
            and torch.autograd.forward_ad._current_level < 0):
        return native().add_rmsnorm_fwd(x, add, weight, eps)
    x = x + add
    return x, rms_norm(x, weight, eps)


def rms_norm_fork(x: torch.Tensor, weight: torch.Tensor, eps: float, centred: bool = False,
                  live: torch.Tensor | None = None) -> tuple[torch.Tensor, torch.Tensor]:
    """``(rms_norm(x), x)`` for a pre-norm block: the second result is the residual branch."""
    if _norm_native(x) and torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad):
        return _RMSNormFn.apply(x, weight, eps, centred, True, live)
    return rms_norm(x, weight, eps, centred, live), x


class _Eagle3InputFn(torch.autograd.Function):
    """``cat([rmsnorm(embeds; w_e), rmsnorm(hidden; w_h)], -1)`` written by two
    strided launches into one [T, 2H] buffer (no separate concat copy)."""

    @staticmethod
    def forward(ctx, embeds, hidden, w_e, w_h, eps, live):
        T, H = hidden.shape
        out = torch.empty((T, 2 * H), dtype=hidden.dtype, device=hidden.device)
        rs_e = torch.empty(T, dtype=torch.float32, device=hidden.device)
        rs_h = torch.empty(T, dtype=torch.float32, device=hidden.device)
        nat = native()
        nat.rmsnorm_fwd(embeds, w_e, None, out[:, :H], rs_e, eps, live)
        nat.rmsnorm_fwd(hidden, w_h, None, out[:, H:], rs_h, eps, live)
        ctx.save_for_backward(embeds, hidden, w_e, w_h, rs_e, rs_h, live)
        ctx.set_materialize_grads(False)
        # second result: the normalised-hidden half on its own, so that a consumer of just
        # that half (the residual branch) hands its gradient back as [T, H] instead of
        # autograd padding it to [T, 2H] (zero fill + copy + add)
        return out, out[:, H:]

    @staticmethod
    def backward(ctx, dout, dhalf):
        embeds, hidden, w_e, w_h, rs_e, rs_h, live = ctx.saved_tensors
        T, H = hidden.shape
        if dout is None:
            dout = torch.zeros((T, 2 * H), dtype=hidden.dtype, device=hidden.device)
        dout = _grad_rows(dout, 2 * H)
        need_e, need_h, need_we, need_wh = ctx.needs_input_grad[:4]
        d_e, dw_e = _norm_backward(dout[:, :H], None, embeds, w_e, rs_e, None, need_e, need_we, False, live)
        d_h, dw_h = _norm_backward(dout[:, H:], _grad_rows(dhalf, H), hidden, w_h, rs_h, None, need_h, need_wh, False, live)
        return d_e, d_h, dw_e, dw_h, None, None


def eagle3_input_concat(embeds, hidden, w_embed_norm, w_hidden_norm, eps, return_hidden_half: bool = False, live: torch.Tensor | None = None):
    """First-layer input of an EAGLE-3 draft: both halves normalised, concatenated
    (``[T, 2H]``).  With ``return_hidden_half`` also returns the normalised-hidden half
    ``[T, H]`` as a result of its own (a view of the first on CUDA)."""
    if _use_native(hidden):
        out, half = _Eagle3InputFn.apply(embeds.contiguous(), hidden.contiguous(), w_embed_norm, w_hidden_norm, eps, live)
    else:
        out = torch.cat([_rms_norm_ref(embeds, w_embed_norm, eps), _rms_norm_ref(hidden, w_hidden_norm, eps)], dim=-1)
        half = out[:, hidden.shape[-1]:]
    return (out, half) if return_hidden_half else out


# --------------------------------------------------------------------------- swiglu
class _SwiGLUFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate_up, live):
        ctx.save_for_backward(gate_up, live)
        return native().swiglu_fwd(gate_up, live)

    @staticmethod
    def backward(ctx, dh):
        gate_up, live = ctx.saved_tensors
        return _settled(native().swiglu_bwd_rows(dh.contiguous(), gate_up, live), live), None


class _GateUpSwiGLUFn(torch.autograd.Function):
    """``h = silu(x @ Wg.T) * (x @ Wu.T)`` with ``W = [Wg; Wu]``: one GEMM whose epilogue stores the
    gate | up product (saved for the backward pass) and the activated product."""

    @staticmethod
    def forward(ctx, x2, weight, use, live):
        gate_up, h = native().gemm_swiglu(x2, weight, gemm_status(x2.device), live)
        ctx.save_for_backward(x2, weight, gate_up, live)
        ctx.use = use
        return h

    @staticmethod
    def backward(ctx, dh):
        x2, weight, gate_up, live = ctx.saved_tensors
        dgu = native().swiglu_bwd_rows(dh.contiguous(), gate_up, live)
        dx, dw = _linear_backward(x2, weight, (None, None), ctx.use, dgu, ctx.needs_input_grad[0], ctx.needs_input_grad[1], live)
        return dx, dw, None, None


def fused_swiglu_enabled() -> bool:
    import os

    return os.environ.get("SB200_FUSED_SWIGLU", "1") != "0"


def linear_swiglu(x: torch.Tensor, weight: torch.Tensor, live: torch.Tensor | None = None) -> torch.Tensor | None:
    """``swiglu(linear(x, weight))`` for a stacked ``[gate; up]`` weight in one launch: the
    activation is formed in the GEMM's epilogue from the accumulator (``SB200_FUSED_SWIGLU=0``
    switches it off).  ``None`` when the operands do not suit the kernel (other dtype or device,
    intermediate size not a multiple of 128) and the caller should run the two steps."""
    x2 = x.reshape(-1, x.shape[-1])
    if (not own_gemm_enabled() or not fused_swiglu_enabled() or not _gemm_operand_ok(x2) or not _gemm_operand_ok(weight)
            or weight.shape[0] % 256 or weight.shape[1] != x2.shape[1]):
        return None
    use = _note_use(weight, None, None) if weight.requires_grad and torch.is_grad_enabled() else None
    h = _GateUpSwiGLUFn.apply(x2, weight, use, live)
    return h.view(*x.shape[:-1], h.shape[-1])


def swiglu(gate_up: torch.Tensor, live: torch.Tensor | None = None) -> torch.Tensor:
    """``silu(gate) * up`` where ``gate_up = [gate | up]`` along the last dim."""
    if _use_native(gate_up):
        shape = gate_up.shape
        out = _SwiGLUFn.apply(gate_up.reshape(-1, shape[-1]).contiguous(), live)
        return out.view(*shape[:-1], shape[-1] // 2)
    gate, up = gate_up.chunk(2, dim=-1)
    return F.silu(gate) * up


# --------------------------------------------------------------------------- rope
def _rope_ref(x, positions, cos_t, sin_t, heads, hd, rot, sign):
    T = x.shape[0]
    xv = x[:, : heads * hd].reshape(T, heads, hd)
    pos = positions.clamp(0, cos_t.shape[0] - 1)
    c = cos_t[pos].unsqueeze(1).to(torch.float32)
    s = (sin_t[pos] * sign).unsqueeze(1).to(torch.float32)
    half = rot // 2
    x1 = xv[..., :half].float()
    x2 = xv[..., half:rot].float()
    y = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s, xv[..., rot:].float()], dim=-1).to(x.dtype)
    return torch.cat([y.reshape(T, heads * hd), x[:, heads * hd :]], dim=-1)


def _unrotate(dq, dk, dv, positions, cos_t, sin_t, heads, hd, rot, live=None):
    """Gradient of a rotation: the ``[T, .]`` gradients side by side in a fresh buffer (an incoming one may be shared with
    other consumers), the first ``heads`` heads rotated back."""
    parts = [_grad_rows(d, math.prod(d.shape[1:])) if d is not None else None for d in (dq, dk, dv)]
    merge = rot % 16 == 0 and all(p is None or (p.shape[1] % hd == 0 and p.data_ptr() % 16 == 0) for p in parts)
    nq = parts[0].shape[1] // hd
    rotate_k = heads > nq
    if merge and heads == nq + (parts[1].shape[1] // hd if rotate_k else 0) and positions.is_contiguous():
        return native().rope_merge(*parts, rotate_k, positions, cos_t, sin_t, hd, rot, -1.0, live)
    d = parts[0].clone() if dk is None else torch.cat([p for p in parts if p is not None], dim=-1)
    native().rope_(d, positions, cos_t, sin_t, heads, hd, rot, -1.0, live)
    return d


class _RopeFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, positions, cos_t, sin_t, heads, hd, rot):
        ctx.save_for_backward(positions, cos_t, sin_t)
        ctx.cfg = (heads, hd, rot)
        native().rope_(x.view(x.shape[0], -1), positions, cos_t, sin_t, heads, hd, rot, 1.0)
        ctx.mark_dirty(x)
        return x

    @staticmethod
    def backward(ctx, dx):
        return _unrotate(dx, None, None, *ctx.saved_tensors, *ctx.cfg).view(dx.shape), None, None, None, None, None, None


def rope_(x, positions, cos_t, sin_t, heads: int, hd: int, rot: int):
    """Neox rotary embedding of the first ``heads`` heads of every row of ``x``
    (``[T, >= heads*hd]`` or ``[T, heads, hd]``), rotating the first ``rot`` channels of each head.
    In place on CUDA; returns the rotated tensor."""
    if _use_native(x):
        if x._is_view() or x.stride(-1) != 1 or (x.dim() == 3 and not x.is_contiguous()):  # noqa: SLF001
            # rotating a view in place would rewrite its base's history (and is refused outright for
            # views that custom functions hand out): work on a private copy instead
            x = x.clone(memory_format=torch.contiguous_format)
        return _RopeFn.apply(x, positions, cos_t, sin_t, heads, hd, rot)
    return _rope_ref(x.reshape(x.shape[0], -1), positions, cos_t, sin_t, heads, hd, rot, 1.0).view(x.shape)


class _RopeSplitFn(torch.autograd.Function):
    """Rotate the q|k heads of a fused projection buffer in place and hand out the
    q / k / v column blocks as views.  Backward lays the three gradients side by side in one
    fresh buffer and un-rotates them on the way, in one pass."""

    @staticmethod
    def forward(ctx, qkv, positions, cos_t, sin_t, heads, hd, rot, nq, nk, live):
        ctx.save_for_backward(positions, cos_t, sin_t, live)
        ctx.cfg = (heads, hd, rot)
        qkv = qkv.detach()
        native().rope_(qkv, positions, cos_t, sin_t, heads, hd, rot, 1.0, live)
        q, k, v = qkv[:, :nq], qkv[:, nq : nq + nk], qkv[:, nq + nk :]
        return q, k, v

    @staticmethod
    def backward(ctx, dq, dk, dv):
        *tables, live = ctx.saved_tensors
        return _settled(_unrotate(dq, dk, dv, *tables, *ctx.cfg, live), live), None, None, None, None, None, None, None, None, None


# --------------------------------------------------------------------------- per-head norms and rotation
def _is_split(block: int, nb: int, split) -> bool:
    """Queries (the first of two rotated blocks) stay whole."""
    return split is not None and not (block == 0 and nb)


def _head_blocks(blocks, split):
    nb = blocks[1] is not None
    return tuple(x for i, b in enumerate(blocks) if b is not None for x in ((b[:split], b[split:]) if _is_split(i, nb, split) else (b,)))


class _NormRopeHeadsFn(torch.autograd.Function):
    """Head norms and rotation of a projection ``[a heads | b heads | plain heads]``; see ``norm_rope_heads``."""

    @staticmethod
    def forward(ctx, src, w_a, w_b, positions, cos_t, sin_t, eps, heads, hd, rot, split, repeated, live):
        na, nb, nv = heads
        src = src.detach()
        out, rstd = native().heads_fwd(src, w_a, na, w_b, nb, eps, positions, cos_t, sin_t, hd, rot, repeated, live)
        ctx.save_for_backward(src, w_a, w_b, rstd, positions, cos_t, sin_t, live)
        ctx.cfg = (heads, hd, rot, split, repeated)
        ctx.set_materialize_grads(False)
        blocks = [out[:, : na * hd], out[:, na * hd :], src[:, (na + nb) * hd : (na + nb + nv) * hd]]
        blocks = [b.unflatten(1, (n, hd)) if n else None for b, n in zip(blocks, heads)]
        if repeated:
            v = blocks[2]
            return blocks[0], blocks[1][:split], blocks[1][split:], v[:split], v[split : split + 1].expand(out.shape[0] - split, nv, hd)
        return _head_blocks(blocks, split)

    @staticmethod
    def backward(ctx, *grads):
        src, w_a, w_b, rstd, positions, cos_t, sin_t, live = ctx.saved_tensors
        (na, nb, nv), hd, rot, split, repeated = ctx.cfg
        it = iter(grads)
        rows = []  # gradients of rows below and from the split on, for each of the three blocks
        for block, n in enumerate((na, nb, nv)):
            for half in range(2):
                g = next(it) if n and half < (2 if _is_split(block, nb, split) else 1) else None
                rows.append(_grad_rows(g, n * hd) if g is not None and g.shape[0] else None)
        dw_a, acc_a, flat_a = _param_grad_target(w_a) if ctx.needs_input_grad[1] else (None, False, False)
        dw_b, acc_b, flat_b = _param_grad_target(w_b) if nb and ctx.needs_input_grad[2] else (None, False, False)
        d = native().heads_bwd(rows, src.shape[0] if split is None else split, src, rstd, w_a, na, w_b, nb, nv, dw_a, acc_a, dw_b, acc_b, positions, cos_t, sin_t, hd, rot, repeated, live)
        return _settled(d, live), None if flat_a else dw_a, None if flat_b else dw_b, None, None, None, None, None, None, None, None, None, None


def norm_rope_heads(src: torch.Tensor, w_a, w_b, eps: float, positions, cos_t, sin_t, heads: tuple[int, int, int], hd: int, rot: int,
                    split: int | None = None, repeated: bool = False, live: torch.Tensor | None = None):
    """Per-head RMSNorm (weights ``w_a``, ``w_b``) and rotary embedding of the first ``heads[0]`` and next ``heads[1]`` heads of
    a projection ``[T, sum(heads) * hd]``; the last ``heads[2]`` heads pass through.  Returns a ``[T, n, hd]`` tensor for every
    block that has heads, or with ``split`` two (rows below it, rows from it on) for every block but the queries, the first of
    two rotated ones.  One launch each way on CUDA (head
    dims 64, 128, 256); the gradients of all results are gathered into one buffer of the projection's layout.

    ``repeated``: ``src`` holds ``split + 2`` rows, and every row from ``split`` on (``positions`` has them all) stands for row
    ``split`` at its own position, as ``repeat_rows`` would lay them out."""
    na, nb, nv = heads
    if repeated and not (nb and nv and _norm_native(src)):
        src, repeated = repeat_rows(src, positions.shape[0]), False
    if (_use_native(src) and src.dtype == torch.bfloat16 and hd in (64, 128, 256) and rot % 16 == 0 and rot <= hd and src.stride(-1) == 1
            and src.stride(0) % 8 == 0 and src.data_ptr() % 16 == 0 and positions.is_contiguous() and all(w is None or w.dtype == src.dtype for w in (w_a, w_b))):
        return _NormRopeHeadsFn.apply(src, w_a, w_b, positions, cos_t, sin_t, eps, heads, hd, rot, split, repeated, live)
    if repeated:
        src = repeat_rows(src, positions.shape[0])
    T, blocks, col = src.shape[0], [], 0
    for n, w in ((na, w_a), (nb, w_b), (nv, None)):
        x = src[:, col : col + n * hd].reshape(T, n, hd) if n else None
        col += n * hd
        if n and w is not None:
            x = rope_(rms_norm(x, w, eps).reshape(T, n * hd), positions, cos_t, sin_t, n, hd, rot).view(T, n, hd)
        blocks.append(x)
    return _head_blocks(blocks, split)


# --------------------------------------------------------------------------- rows that a step needs
class StepRows(NamedTuple):
    """Rows of a packed batch that a training-time-test step needs, and what its passes read of them (``step_rows``).

    A tensor "of the rows" has one row per listed row of the batch and as many rows in all as the batch, of which the first
    ``live`` are in use: shapes do not depend on the mask, and the count stays on the device."""

    index: torch.Tensor  # int64 [T]: the batch's row
    inverse: torch.Tensor  # int32 [T]: where a row of the batch is listed, -1: nowhere
    live: torch.Tensor  # int32 [1]
    target_index: torch.Tensor  # the same for the verifier's rows
    target_live: torch.Tensor
    ids: torch.Tensor  # int64 [passes, T], shifted by the pass
    positions: torch.Tensor
    mask: torch.Tensor  # bool [passes, T]
    prev_correct: torch.Tensor  # bool [T]
    target_row: torch.Tensor  # int32 [passes, T]: the verifier's listed row to compare with, -1: none
    intervals: list  # of (lo, hi)
    extra: list  # per pass: None, then int32 [T, pass]


def step_rows(mask: torch.Tensor, ids: torch.Tensor, positions: torch.Tensor, intervals: list, passes: int, targets: bool = True) -> StepRows:
    """Which rows of a packed batch the passes of a training-time-test step need, the batch in their order.

    Pass ``s`` compares row ``t`` with the verifier's row ``t + s`` where ``mask[t + s]`` is set, and follows the rows that
    were right in every pass from where ``mask[t]`` is.  A later pass sees a row's own keys of the passes before and nothing
    else of them, so a row that no comparison reads serves as context keys in pass 0 only.  ``mask`` bool / uint8 ``[T]``,
    ``intervals``: up to two key intervals ``(lo, hi)`` of the rows.  Rows are listed in ascending order; the count is a
    multiple of 256 or all of them (on the CPU exact), filled up with rows that nobody asked for.  Without ``targets`` (labels
    instead of a verifier's rows) ``mask`` and ``ids`` may reach past the rows, of which there are as many as ``positions``."""
    T, N = positions.shape[0], ids.shape[0]
    if _use_native(ids):
        both = [lo._base if lo._base is not None and lo._base is hi._base and lo._base.shape == (2, T) else torch.stack([lo, hi]) for lo, hi in intervals]
        index, inverse, count, ids, positions, mask, prev, target_row, spans, extra = native().step_rows(mask.contiguous(), ids.contiguous(), positions.contiguous(), both, passes, targets)
        offsets = [T * s * (s - 1) // 2 for s in range(passes)]
        extra = [None] + [extra.view(-1)[offsets[s] : offsets[s] + T * s].view(T, s) for s in range(1, passes)]
        return StepRows(index[0], inverse[0], count[:1], index[1], count[1:], ids, positions, mask, prev, target_row, [(s[0], s[1]) for s in spans], extra)
    m = torch.cat([mask.bool(), torch.zeros(passes, dtype=torch.bool)])
    lists = []
    for wanted in (torch.stack([m[s : s + T] for s in range(passes)]).any(0),
                   torch.stack([torch.cat([torch.zeros(s, dtype=torch.bool), m[: T - s]]) for s in range(passes) if s < T]).any(0) & targets):
        at = wanted.nonzero().view(-1)
        inverse = torch.full((T,), -1, dtype=torch.int32)
        inverse[at] = torch.arange(at.numel(), dtype=torch.int32)
        lists.append((torch.cat([at, at.new_zeros(T - at.numel())]), inverse, torch.tensor([at.numel()], dtype=torch.int32)))
    (index, inverse, live), (target_index, target_inverse, target_live) = lists
    on = torch.arange(T) < live
    u = index + torch.arange(passes)[:, None]
    there = on & (u < N)
    u = u.clamp(max=N - 1)
    zero = torch.zeros((), dtype=torch.long)
    extra = [None] + [torch.where(on[:, None], torch.arange(s, dtype=torch.int32) * T + torch.arange(T, dtype=torch.int32)[:, None], -1) for s in range(1, passes)]
    return StepRows(index, inverse, live, target_index, target_live, torch.where(there, ids[u], zero),
                    torch.where(on, positions[index] + torch.arange(passes)[:, None], zero), there & m[u], on & m[index],
                    torch.where(there, target_inverse[u.clamp(max=T - 1)], -1), [tuple(torch.where(on, v[index], 0) for v in pair) for pair in intervals], extra)


class _TakeRowsFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, index, inverse, live, *xs):
        ctx.save_for_backward(inverse)
        ctx.set_materialize_grads(False)
        return tuple(native().take_rows(xs, index, live))

    @staticmethod
    def backward(ctx, *ds):
        (inverse,) = ctx.saved_tensors
        given = [i for i, d in enumerate(ds) if d is not None and ctx.needs_input_grad[3 + i]]
        grads = iter(native().put_rows([_grad_rows(ds[i], ds[i].shape[1]) for i in given], inverse)) if given else None
        return None, None, None, *(next(grads) if i in given else None for i in range(len(ds)))


def take_rows(index: torch.Tensor, inverse: torch.Tensor, live: torch.Tensor, *xs: torch.Tensor) -> tuple[torch.Tensor, ...]:
    """Rows ``index`` of one or two matrices ``[T, W]``, as ``step_rows`` lists them; the rows from ``live`` on are not written
    (zero on the CPU).  The gradient is a row copy, zero where a row was not taken."""
    if _use_native(index):
        return _TakeRowsFn.apply(index, inverse, live, *(_grad_rows(x, x.shape[1]) for x in xs))
    return tuple(only_live(x[index], live) for x in xs)


def rms_norm_taken(x: torch.Tensor, weight: torch.Tensor, eps: float, index: torch.Tensor, live: torch.Tensor) -> torch.Tensor:
    """``rms_norm`` of the rows ``index`` of ``x``, where nothing is differentiated."""
    if _norm_native(x):
        if torch.autograd.forward_ad._current_level >= 0 or torch._C._are_functorch_transforms_active():  # noqa: SLF001
            rms_norm(x, weight, eps)  # for its refusal: a tangent or a batch dimension would get lost in a bare kernel call
        y = torch.empty((index.shape[0], x.shape[1]), dtype=x.dtype, device=x.device)
        native().norm_fwd(_grad_rows(x, x.shape[1]), weight, index, y, None, eps, False, live)
        return y
    return rms_norm(only_live(x[index], live), weight, eps)


# --------------------------------------------------------------------------- repeated rows, embedding
class _RepeatRowsFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, n):
        T = x.shape[0] - 2
        out = torch.empty((n, x.shape[1]), dtype=x.dtype, device=x.device)
        out[:T] = x[:T]
        out[T:] = x[T]
        ctx.T = T
        return out

    @staticmethod
    def backward(ctx, d):
        T = ctx.T
        dx = torch.empty((T + 2, d.shape[1]), dtype=d.dtype, device=d.device)
        dx[:T] = d[:T]
        native().repeated_rows_sum(_grad_rows(d[T:], d.shape[1]), dx[T:])
        return dx, None


def repeat_rows(x: torch.Tensor, n: int) -> torch.Tensor:
    """``[T + 2, W] -> [n, W]``: the first ``T`` rows, then row ``T`` as often as it takes (``n > T``).  The last two rows of
    ``x`` hold the same values; a gradient reaches them as the rounded sum over the repeated rows and the rest that rounding
    left, so products with the two keep the sum at twice the precision of bf16."""
    T = x.shape[0] - 2
    if _use_native(x) and x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0 and torch.is_grad_enabled() and x.requires_grad:
        return _RepeatRowsFn.apply(x, n)
    return torch.cat([x[:T], x[T : T + 1].expand(n - T, -1)])


class _EmbeddingFn(torch.autograd.Function):
    """Rows of ``weight``; the gradient goes straight into the engine's flat buffer (a dense one of autograd's own was zeroed,
    filled and then added to it: 3.7 GB of traffic for a 152k x 4096 table), duplicates summed in fp32 in a fixed order."""

    @staticmethod
    def forward(ctx, ids, weight, padding_idx):
        ctx.save_for_backward(ids, weight)
        ctx.padding_idx = padding_idx
        return F.embedding(ids, weight)

    @staticmethod
    def backward(ctx, d):
        ids, weight = ctx.saved_tensors
        dw, accumulate, attached = _param_grad_target(weight)
        if not accumulate:
            dw.zero_()
        order = torch.sort(ids, stable=True)
        native().embedding_bwd(order.values, order.indices, _grad_rows(d, d.shape[1]), -1 if ctx.padding_idx is None else ctx.padding_idx, dw, accumulate)
        return None, None if attached else dw, None


def embedding(ids: torch.Tensor, weight: torch.Tensor, padding_idx: int | None = None) -> torch.Tensor:
    """``F.embedding`` of flat ``ids`` for a table that is trained."""
    if (_use_native(weight) and weight.dtype == torch.bfloat16 and weight.requires_grad and torch.is_grad_enabled() and weight.shape[1] % 8 == 0
            and ids.dtype == torch.int64):
        return _EmbeddingFn.apply(ids.reshape(-1), weight, padding_idx)
    return F.embedding(ids, weight, padding_idx)


# --------------------------------------------------------------------------- gated attention
class _SplitGatedQueryFn(torch.autograd.Function):
    """``(centred_rms_norm(qg[..., :hd]), qg[..., hd:])``; the query half is read and its gradient written in place inside the
    ``[T, heads, 2 * hd]`` buffer, into the other half of which ``_GatedFn`` has put the gate's gradient."""

    @staticmethod
    def forward(ctx, qg, weight, eps, live):
        T, heads, two = qg.shape
        hd = two // 2
        x2 = qg.view(T * heads, two)[:, :hd]
        q = torch.empty((T, heads, hd), dtype=qg.dtype, device=qg.device)
        rstd = torch.empty(T * heads, dtype=torch.float32, device=qg.device)
        native().norm_fwd(x2, weight, None, q.view(T * heads, hd), rstd, eps, True, live)
        ctx.save_for_backward(qg, weight, rstd, live)
        return q, qg[..., hd:]

    @staticmethod
    def backward(ctx, dq, dgate):
        qg, weight, rstd, live = ctx.saved_tensors
        T, heads, two = qg.shape
        hd = two // 2
        in_place = (dgate.dtype == qg.dtype and dgate.stride() == (heads * two, two, 1) and dgate.storage_offset() == hd
                    and dgate.untyped_storage().nbytes() == qg.numel() * qg.element_size())
        if in_place:
            d = dgate.as_strided(qg.shape, (heads * two, two, 1), 0)
        else:
            d = torch.empty_like(qg)
            d[..., hd:] = dgate
        rows = T * heads
        dw, accumulate, attached = _param_grad_target(weight) if ctx.needs_input_grad[1] else (None, False, False)
        native().rmsnorm_bwd(_grad_rows(dq, hd), None, qg.view(rows, two)[:, :hd], weight, rstd, None, d.view(rows, two)[:, :hd], dw, accumulate, True, live)
        return _settled(d.view(rows, two), live).view(qg.shape), None if attached else dw, None, None


class _GatedFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, out, gate, live):
        ctx.save_for_backward(out, gate, live)
        return native().gate_mul_fwd(out, gate)

    @staticmethod
    def backward(ctx, dy):
        out, gate, live = ctx.saved_tensors
        T, heads, hd = out.shape
        dgate = torch.empty((T, heads, gate.stride(1)), dtype=out.dtype, device=out.device)[..., -hd:]  # of a projection: its second half
        return _settled(native().gate_mul_bwd(dy.contiguous(), out, gate, dgate), live), _settled(dgate, live), None


def split_gated_query(qg: torch.Tensor, weight: torch.Tensor, eps: float, live: torch.Tensor | None = None):
    """Query and gate of a gated attention from the ``[T, heads, 2 * hd]`` projection: the query normalised with a zero-centred
    weight, the gate as a view (``live``: heads in use, of all tokens).  ``None`` where the kernels do not take the tensor and the caller runs the steps one by one."""
    if not (_norm_native(qg) and qg.is_contiguous() and qg.shape[-1] % 16 == 0):
        return None
    return _SplitGatedQueryFn.apply(qg, weight, eps, live)


def gated(out: torch.Tensor, gate: torch.Tensor, live: torch.Tensor | None = None) -> torch.Tensor:
    """``out * sigmoid(gate)`` for ``[T, heads, hd]`` CUDA tensors, ``gate`` as ``split_gated_query`` returns it (``live``: tokens
    in use; the kernels run over all)."""
    return _GatedFn.apply(out.contiguous(), gate, live)


def rope_split(qkv, positions, cos_t, sin_t, heads: int, hd: int, rot: int, nq: int, nk: int, live: torch.Tensor | None = None,
               unseen: bool = False):
    """``rope_`` on the first ``heads`` heads of ``qkv`` ([T, nq + nk + nv]) followed by
    the split into ``(q [T, nq], k [T, nk], v [T, rest])``.  On CUDA the buffer is
    rotated in place and the results are views of it: the caller must own ``qkv``
    (a fresh projection output) and must not modify the views in place.  ``unseen``: nobody else holds it either, so that it is
    rotated in place without a gradient too (else a view is copied first)."""
    if _use_native(qkv) and qkv.requires_grad and torch.is_grad_enabled():
        return _RopeSplitFn.apply(qkv, positions, cos_t, sin_t, heads, hd, rot, nq, nk, live)
    if unseen and _use_native(qkv) and not torch.is_grad_enabled() and qkv.dim() == 2 and qkv.stride(-1) == 1 and torch.autograd.forward_ad._current_level < 0:
        out = qkv.detach()  # (``rope_`` would work on a copy of a view)
        native().rope_(out, positions, cos_t, sin_t, heads, hd, rot, 1.0, live)
        return out[:, :nq], out[:, nq : nq + nk], out[:, nq + nk :]
    out = rope_(qkv, positions, cos_t, sin_t, heads, hd, rot)
    return out[:, :nq], out[:, nq : nq + nk], out[:, nq + nk :]


# --------------------------------------------------------------------------- losses
def _row_loss_ref(op: str, logits, targets):
    """fp32 per-row loss and both argmaxes (``logits``/``targets``: [rows, V])."""
    lq = torch.log_softmax(logits.float(), dim=-1)
    lp = torch.log_softmax(targets.float(), dim=-1)
    if op == "kl_div":
        p = lp.exp()
        loss = torch.where(p > 0, p * (lp - lq), torch.zeros_like(p)).sum(-1)
    elif op == "rkl":
        q = lq.exp()
        loss = torch.where(q > 0, q * (lq - lp), torch.zeros_like(q)).sum(-1)
    elif op == "jsd":
        lm = torch.logaddexp(lq, lp) - 0.6931471805599453
        p, q = lp.exp(), lq.exp()
        loss = 0.5 * ((p * (lp - lm)).sum(-1) + (q * (lq - lm)).sum(-1))
    elif op == "ce":
        loss = -lq.gather(-1, targets.argmax(-1, keepdim=True)).squeeze(-1)
    elif op == "tv":
        loss = 1.0 - torch.minimum(lq.exp(), lp.exp()).sum(-1)
    else:
        raise ValueError(f"unknown loss op {op!r}")
    return loss


class _RowLossFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets, op, shift, rows, active, target_row=None, with_tv=False):
        loss, stats, am_d, am_t, tv = native().loss_fwd_tv(op, logits, targets, active, None, shift, rows, target_row, with_tv)
        ctx.save_for_backward(logits, targets, stats, target_row)
        ctx.cfg = (op, shift, rows)
        out = (am_d, am_t, tv) if with_tv else (am_d, am_t)
        ctx.mark_non_differentiable(*out)
        return loss, *out

    @staticmethod
    def backward(ctx, dloss, *_):
        logits, targets, stats, target_row = ctx.saved_tensors
        op, shift, rows = ctx.cfg
        d = native().loss_bwd_scaled(op, logits, targets, dloss.contiguous().float(), None, stats, shift, rows, target_row)
        return d, None, None, None, None, None, None, None


class _LmHeadLossFn(torch.autograd.Function):
    """``fused_row_loss(op, hidden @ weight.T, targets, shift, rows, active)`` with the head's GEMM
    and the forward reduction of the loss in one kernel: the logits tile is reduced to
    online-softmax records while it is still in tensor memory, so the forward never re-reads
    ``[T, V]`` logits and targets.  The logits are stored (bf16) for the backward pass, which is
    the row-loss backward kernel followed by the input-gradient GEMM."""

    @staticmethod
    def forward(ctx, hidden, weight, targets, op, shift, rows, active, use):
        logits, loss, stats, am_d, am_t = native().lmhead_loss_fwd(op, hidden, weight, targets, active, shift, rows, gemm_status(hidden.device))
        ctx.save_for_backward(hidden, weight, targets, logits, stats)
        ctx.cfg, ctx.use = (op, shift, rows), use
        ctx.mark_non_differentiable(am_d, am_t)
        return loss, am_d, am_t

    @staticmethod
    def backward(ctx, dloss, _a, _b):
        hidden, weight, targets, logits, stats = ctx.saved_tensors
        op, shift, rows = ctx.cfg
        d = native().loss_bwd(op, logits, targets, dloss.contiguous().float(), stats, shift, rows)
        dx, dw = _linear_backward(hidden, weight, (None, None), ctx.use, d, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        return dx, dw, None, None, None, None, None, None


FUSED_HEAD_OPS = ("kl_div", "ce")


def fused_head_enabled() -> bool:
    import os

    return os.environ.get("SB200_FUSED_HEAD", "0") == "1"


def lm_head_loss_ok(op: str, hidden: torch.Tensor, weight: torch.Tensor, targets: torch.Tensor) -> bool:
    """Whether the fused head of ``lm_head_loss_raw`` applies and is switched on."""
    return (op in FUSED_HEAD_OPS and fused_head_enabled() and own_gemm_enabled()
            and _gemm_operand_ok(hidden) and _gemm_operand_ok(weight) and _gemm_operand_ok(targets)
            and weight.shape[0] % 8 == 0 and hidden.shape[0] > 128)


def lm_head_loss_raw(op: str, hidden: torch.Tensor, weight: torch.Tensor, targets: torch.Tensor, shift: int, rows: int, active):
    """Per-row loss between ``(hidden @ weight.T)[r]`` and ``targets[r + shift]`` for ``r < rows``
    plus both argmaxes (int32), like ``fused_row_loss_raw`` on the product; ``None`` when the
    fused head does not apply (other loss, other dtype / layout, not switched on) and the caller
    should form the logits itself.  Opt-in (``SB200_FUSED_HEAD=1``): at 2048 x 32000 x 4096 the
    fused kernel measured 0.466 ms against 0.443 ms for the GEMM followed by the row-loss
    kernel (its statistics epilogue holds the tensor pipe at 70 % active against 88 % for the
    plain store epilogue), so the two-kernel form is the default."""
    if not lm_head_loss_ok(op, hidden, weight, targets):
        return None
    use = _note_use(weight, None, None) if weight.requires_grad and torch.is_grad_enabled() else None
    return _LmHeadLossFn.apply(hidden, weight, targets, LOSS_OPS[op], shift, rows, active, use)


class _StepTailFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, row_loss, pred, target, mask, prev, decay, eps):
        out, weight, _ = native().step_tail(row_loss, pred, target, mask, prev, decay, eps, None)
        out = out[:4]
        ctx.save_for_backward(weight)
        ctx.mark_dirty(prev)
        ctx.mark_non_differentiable(prev)
        return out, prev

    @staticmethod
    def backward(ctx, dout, _dprev):
        (weight,) = ctx.saved_tensors
        return weight * dout[0], None, None, None, None, None, None


class _StepLossFn(torch.autograd.Function):
    """Row loss and tail of one training-time-test pass: two launches forward, one backward.  As separate functions autograd
    put a zero fill in front of every result that is not differentiated, and a copy and a product around the loss itself:
    fourteen launches more in each pass, on steps whose kernels take 2 us."""

    @staticmethod
    def forward(ctx, logits, targets, earlier, op, shift, rows, mask, prev, decay, eps, target_row, live):
        row_loss, stats, pred, tgt = native().loss_fwd_either(op, logits, targets, mask, prev, shift, rows, target_row)
        out, weight, total = native().step_tail(row_loss, pred, tgt, mask, prev, decay, eps, earlier, target_row)
        ctx.save_for_backward(logits, targets, stats, weight, target_row, live)
        ctx.cfg = (op, shift, rows)
        ctx.mark_non_differentiable(out)
        ctx.set_materialize_grads(False)
        return total, out

    @staticmethod
    def backward(ctx, dtotal, _dout):
        if dtotal is None:
            return (None,) * 12
        logits, targets, stats, weight, target_row, live = ctx.saved_tensors
        op, shift, rows = ctx.cfg
        d = native().loss_bwd_scaled(op, logits, targets, weight, dtotal.float(), stats, shift, rows, target_row, live)
        return _settled(d, live), None, dtotal if ctx.needs_input_grad[2] else None, None, None, None, None, None, None, None, None, None


def ttt_step_loss(op: str, logits, targets, earlier, shift: int, rows: int, mask, prev_correct, decay: float, eps: float, target_row=None, live=None):
    """``fused_row_loss_raw`` over the rows marked in ``mask`` or ``prev_correct`` followed by ``ttt_step_tail`` (CUDA, bf16
    logits).  Returns ``(earlier + loss, out)`` with ``out`` = loss, correct, total, cond_total, 1; ``earlier``: the loss of
    the passes before or ``None``; the loss itself is differentiable through the first result.  ``target_row`` (int32
    ``[rows]``): the row of ``targets`` to compare with in place of ``shift``, -1 for none (``step_rows``)."""
    if not _use_native(logits):
        there = torch.ones(rows, dtype=torch.bool) if target_row is None else target_row >= 0
        mask, was = mask[:rows].bool() & there, prev_correct[:rows] & there
        tg = targets[shift : shift + rows] if target_row is None else targets[target_row.clamp(min=0).long()]
        row_loss, pred, tgt = fused_row_loss(op, logits[:rows], tg, active=mask | was)
        out = ttt_step_tail(row_loss, pred, tgt, mask, was, decay, eps)
        prev_correct[:rows] = torch.where(there, was, prev_correct[:rows])
        total = out[0] if earlier is None else earlier + out[0]
        return total, torch.cat([out.detach(), out.new_ones(1)])
    logits, targets = (t if t.stride(-1) == 1 else t.contiguous() for t in (logits, targets))
    return _StepLossFn.apply(logits, targets, earlier, LOSS_OPS[op], shift, rows, mask, prev_correct, float(decay), float(eps), target_row, live)


def ttt_step_tail(row_loss, pred_ids, target_ids, mask, prev_correct, decay: float, eps: float):
    """Masked-mean loss of one training-time-test pass and its accuracy counters.

    ``row_loss`` fp32 ``[rows]`` (differentiable), ``pred_ids`` / ``target_ids`` integer
    ``[rows]``, ``mask`` bool / uint8 ``[rows]``, ``prev_correct`` bool / uint8 ``[>= rows]``
    (AND-ed in place with this pass's hits).  Returns fp32 ``[4]``: ``loss =
    decay * sum(row_loss * mask) / (sum(mask) + eps)``, ``correct = sum(prev & hit & mask)``,
    ``total = sum(mask)``, ``cond_total = sum(prev before the update)``.  One launch on
    CUDA; the same arithmetic with torch ops elsewhere."""
    rows = row_loss.shape[0]
    if _use_native(row_loss) and pred_ids.dtype == torch.int32 and target_ids.dtype == torch.int32:
        out, _ = _StepTailFn.apply(row_loss.contiguous(), pred_ids, target_ids, mask, prev_correct, float(decay), float(eps))
        return out
    m = mask[:rows].bool()
    was = prev_correct[:rows].bool()
    cond_total = was.sum().float()
    now = was & (pred_ids[:rows] == target_ids[:rows])
    prev_correct[:rows] = now.to(prev_correct.dtype)
    mf = m.to(row_loss.dtype)
    loss = decay * (row_loss * mf).sum() / (mf.sum() + eps)
    return torch.stack([loss, (now & m).sum().float(), mf.sum().float(), cond_total])


def fused_row_loss_raw(op: str, logits, targets, shift: int, rows: int, active):
    """``fused_row_loss`` on CUDA without the widening of the argmax by-products (int32)."""
    if logits.stride(-1) != 1:
        logits = logits.contiguous()
    if targets.stride(-1) != 1:
        targets = targets.contiguous()
    return _RowLossFn.apply(logits, targets, LOSS_OPS[op], shift, rows, active)


def fused_row_loss(op: str, logits, targets, shift: int = 0, rows: int | None = None, active=None, target_row=None, with_tv: bool = False):
    """Per-row loss between ``logits[r]`` and ``targets[r + shift]`` (``targets[target_row[r]]`` with int32 ``target_row``) for
    ``r < rows``.

    Returns ``(loss[rows] fp32, argmax_logits[rows], argmax_targets[rows])``, and for ``kl_div`` ``with_tv`` also the rows' total
    variation (no gradient).  ``active`` (bool[rows], optional) marks rows worth computing; inactive rows get
    loss 0 and sentinel argmaxes (-1 / -2, never equal).  Gradients flow to
    ``logits`` only; the buffer that comes back has ``logits.shape`` with rows
    ``>= rows`` zeroed.
    """
    if logits.dim() != 2 or targets.dim() != 2:
        raise ValueError("fused_row_loss expects [rows, V] inputs")
    if rows is None:
        rows = logits.shape[0] if target_row is not None else min(logits.shape[0], targets.shape[0] - shift)
    if _use_native(logits):
        if logits.stride(-1) != 1:
            logits = logits.contiguous()
        if targets.stride(-1) != 1:
            targets = targets.contiguous()
        loss, am_d, am_t, *tv = _RowLossFn.apply(logits, targets, LOSS_OPS[op], shift, rows, active, target_row, with_tv)
        return loss, am_d.long(), am_t.long(), *tv
    lg = logits[:rows]
    tg = targets[target_row.long()[:rows]] if target_row is not None else targets[shift : shift + rows]
    loss = _row_loss_ref(op, lg, tg)
    tv = [_row_loss_ref("tv", lg.detach(), tg)] if with_tv else []
    am_d, am_t = lg.argmax(-1), tg.argmax(-1)
    if active is not None:
        act = active.bool()
        loss, *tv = (torch.where(act, v, torch.zeros_like(v)) for v in (loss, *tv))
        am_d = torch.where(act, am_d, torch.full_like(am_d, -1))
        am_t = torch.where(act, am_t, torch.full_like(am_t, -2))
    return loss, am_d, am_t, *tv


class _TokenCEFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, labels, keep, live):
        loss, stats = native().ce_label_fwd(logits, labels, keep)
        ctx.save_for_backward(logits, stats, live)
        return loss

    @staticmethod
    def backward(ctx, dloss):
        logits, stats, live = ctx.saved_tensors
        # the CE backward only needs the saved label (stats[4]) and the draft statistics
        d = native().loss_bwd_scaled(LOSS_OPS["ce"], logits, logits, dloss.contiguous().float(), None, stats, 0, logits.shape[0], None, live)
        return _settled(d, live), None, None, None


def token_cross_entropy(logits: torch.Tensor, labels: torch.Tensor, keep: torch.Tensor | None = None, live: torch.Tensor | None = None) -> torch.Tensor:
    """Per-row cross-entropy of ``logits [n, V]`` against integer ``labels [n]``;
    rows with ``keep == False`` contribute 0 (and no gradient).  ``live``: see ``step_rows``; no row behind it is kept."""
    if _use_native(logits):
        if logits.stride(-1) != 1:
            logits = logits.contiguous()
        keep_b = keep.to(torch.bool).contiguous() if keep is not None else None
        return _TokenCEFn.apply(logits, labels.long().contiguous(), keep_b, live)
    loss = F.cross_entropy(logits.float(), labels.long(), reduction="none")
    return loss if keep is None else torch.where(keep.bool(), loss, torch.zeros_like(loss))


# --------------------------------------------------------------------------- optimizer
def sum_of_squares(flat: torch.Tensor, out: torch.Tensor, accumulate: bool = False) -> torch.Tensor:
    """``out[0] (+)= sum(flat**2)`` in fp32, deterministic two-stage reduction."""
    if _use_native(flat):
        native().sumsq(flat, out, accumulate)
    else:
        s = flat.float().pow(2).sum()
        out[0] = out[0] + s if accumulate else s
    return out


HYPER_LEN = 16


def adamw_step_(master, m, v, grad, w16, hyper, norm_sq=None) -> None:
    """One fused AdamW step over flat buffers.  ``hyper`` (fp32[16], same device):
    lr, beta1, beta2, eps, weight_decay, bias_correction1, bias_correction2,
    max_grad_norm (<= 0 disables clipping), grad_scale.  ``norm_sq`` holds the global
    sum of squared (unscaled) gradients.  ``w16`` (optional) receives the bf16 copy."""
    if _use_native(master):
        native().adamw(master, m, v, grad, w16, hyper, norm_sq)
        return
    lr, b1, b2, eps, wd, bc1, bc2, max_norm, gscale = (float(hyper[i]) for i in range(9))
    if max_norm > 0 and norm_sq is not None:
        coef = max_norm / (gscale * float(norm_sq[0]) ** 0.5 + 1e-6)
        if coef < 1.0:
            gscale *= coef
    g = grad.float() * gscale
    master.mul_(1 - lr * wd)
    m.mul_(b1).add_(g, alpha=1 - b1)
    v.mul_(b2).addcmul_(g, g, value=1 - b2)
    denom = v.sqrt() / (bc2**0.5) + eps
    master.addcdiv_(m, denom, value=-lr / bc1)
    if w16 is not None:
        w16.copy_(master)
