"""Mixture-of-experts layer whose experts all live on one GPU, as one differentiable call.

Routing results in, weighted sum of the experts out: two planning launches, a gather into the padded expert order, two
grouped tcgen05 products (the first forms ``silu(gate) * up`` in its epilogue), one combining launch that also adds the
shared expert and the residual.  The backward pass mirrors it, and the experts' weight gradients go straight into the
training engine's flat buffer.  (Counterpart of the expert loop that the reference takes from its wrapped Hugging Face
modules, src/speculators/models/mtp/model_definitions.py:159-205.)
"""

from __future__ import annotations

import os

import torch

from speculators_b200 import ops

__all__ = ["moe_experts", "moe_experts_ok"]

_MAX_EXPERTS = 1024  # the planning kernels keep a counter per expert in shared memory


def moe_experts_ok(x: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor) -> bool:
    """bf16 CUDA rows, experts as contiguous stacks with widths in whole 256-column tiles of the grouped products."""
    return (x.is_cuda and x.shape[0] > 0 and ops.own_gemm_enabled() and os.environ.get("SB200_MOE_GEMM", "tcgen05") != "library"
            and all(t.dtype == torch.bfloat16 for t in (x, gate_up, down)) and gate_up.is_contiguous() and down.is_contiguous()
            and gate_up.shape[0] <= _MAX_EXPERTS and gate_up.shape[1] % 256 == 0 and gate_up.shape[2] % 256 == 0 and down.shape[2] % 256 == 0)


class _MoEExpertsFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, top_p, top_e, w_gu, w_d, shared, gate, residual, uses, live):
        nat, status = ops.native(), ops.gemm_status(x.device)
        k, E = top_e.shape[1], w_gu.shape[0]
        capacity = (top_e.numel() + 127 * E + 127) // 128 * 128  # worst case: every expert's tail padded by 127 rows
        seg, tiles, slot_row, row_slot = nat.moe_plan(top_e, E, capacity, k, live)
        x_pad = nat.moe_gather(x, row_slot, seg, k)
        gate_up, h = nat.gemm_grouped_swiglu(x_pad, w_gu, seg, tiles, status)
        y_pad = torch.empty((capacity, w_d.shape[1]), dtype=x.dtype, device=x.device)
        nat.gemm_grouped_rows(h, w_d, y_pad, False, seg, tiles, status)
        out = nat.moe_combine(y_pad, slot_row, top_p, shared, gate, residual, live)
        ctx.save_for_backward(x_pad, gate_up, h, y_pad, top_p, w_gu, w_d, shared, gate, seg, tiles, slot_row, row_slot, live)
        ctx.with_residual, ctx.uses = residual is not None, uses
        return out

    @staticmethod
    def backward(ctx, dout):
        x_pad, gate_up, h, y_pad, top_p, w_gu, w_d, shared, gate, seg, tiles, slot_row, row_slot, live = ctx.saved_tensors
        nat, status = ops.native(), ops.gemm_status(dout.device)
        need = ctx.needs_input_grad
        dout = dout.contiguous()
        dy_pad, *grads = nat.moe_combine_bwd(dout, y_pad, row_slot, seg, top_p, shared, gate, live)
        dp, dshared, dgate = (ops._settled(d, live) if d.numel() else d for d in grads)  # noqa: SLF001

        def weight_gradient(needed, dy, rows, w, use):
            if not needed:
                return None
            flat = getattr(w, "_flat_grad", None)
            if flat is None:
                dw = torch.empty_like(w)
                nat.gemm_grouped_wgrad(dy, rows, dw, False, seg, tiles, status)
                return dw

            def launch(uses):
                target, accumulate, _ = ops._param_grad_target(w, beside=True)  # noqa: SLF001
                dys, xs, segs = (list(part) for part in zip(*uses))
                nat.gemm_grouped_wgrad_parts(dys, xs, target, accumulate, segs, tiles, status)

            ops._gather_use(w, ("experts",), use, (dy, rows, seg), launch)  # noqa: SLF001
            return None

        dw_d = weight_gradient(need[4], dy_pad, h, w_d, ctx.uses[1])
        dx = dw_gu = None
        if need[0] or need[3]:
            dh = torch.empty_like(h)
            nat.gemm_grouped_rows(dy_pad, w_d, dh, True, seg, tiles, status)
            dgu = nat.swiglu_bwd_rows(dh, gate_up, seg[-1:])
            dw_gu = weight_gradient(need[3], dgu, x_pad, w_gu, ctx.uses[0])
            if need[0]:
                dx_pad = torch.empty_like(x_pad)
                nat.gemm_grouped_rows(dgu, w_gu, dx_pad, True, seg, tiles, status)
                dx = ops._settled(nat.moe_gather_bwd(dx_pad, slot_row, top_p.shape[1], live), live)  # noqa: SLF001
        with_shared = shared is not None
        return dx, dp, None, dw_gu, dw_d, dshared if with_shared else None, dgate if with_shared else None, dout if ctx.with_residual else None, None, None


def moe_experts(x, top_p, top_e, gate_up, down, shared=None, shared_gate=None, residual=None, live=None) -> torch.Tensor:
    """``sum_j top_p[t, j] * expert_{top_e[t, j]}(x[t]) (+ sigmoid(shared_gate[t]) * shared[t]) (+ residual[t])`` for
    operands that ``moe_experts_ok`` accepts; ``x [T, H]``, ``top_e`` int64 and ``top_p`` of ``x``'s dtype ``[T, k]``,
    ``shared_gate`` ``[T, 1]`` before its sigmoid.  ``live``: tokens in use (``ops.step_rows``); the others go to no expert."""
    def rows(t):
        return None if t is None else t.contiguous()

    grad = torch.is_grad_enabled()
    uses = tuple(ops._note_use(w, "experts") if grad and w.requires_grad else None for w in (gate_up, down))  # noqa: SLF001
    return _MoEExpertsFn.apply(rows(x), rows(top_p), rows(top_e), gate_up, down, rows(shared), rows(shared_gate), rows(residual), uses, live)
