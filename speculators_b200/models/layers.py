"""Decoder building blocks owned by this framework.

The reference assembles its drafts from Hugging Face ``LlamaDecoderLayer`` /
``Qwen3DecoderLayer`` classes (src/speculators/models/base_components.py:39-100).
Here the blocks are written against ``speculators_b200.ops`` so that on a B200
every hot step is one of the package's own kernels, while the parameter *names*
in ``state_dict()`` stay the Hugging Face ones (``self_attn.q_proj.weight``,
``mlp.gate_proj.weight`` ...), which is what the checkpoint format and vLLM
expect.

Projections that share an input are stored fused (q|k|v and gate|up) so each
runs as a single GEMM; ``FusedLinear`` splits / merges them at the
``state_dict`` boundary.
"""

from __future__ import annotations

import math

import torch
from torch import nn

from speculators_b200 import ops
from speculators_b200.layer_config import TransformerLayerConfig
from speculators_b200.ops import AttnSpec

__all__ = [
    "Attention",
    "DecoderLayer",
    "decoder_layer_fwd",
    "FusedLinear",
    "Linear",
    "MLP",
    "NEEDED_ROWS_FROM",
    "RMSNorm",
    "RotaryTable",
    "norm_of_sum",
    "stops_at_count",
    "takes_listed_rows",
    "unobserved",
    "watched",
]


_ROW_MODULES: set[type] = {nn.Embedding}


def stops_at_count(cls: type) -> type:
    """Class decorator: a module of this class runs over the rows in use alone (``live``, ``rows``), or row by row.  A class
    derived from it says so itself or counts as one that reads all rows."""
    _ROW_MODULES.add(cls)
    return cls


def _tree(modules) -> list[nn.Module]:
    """``modules`` and what is below them.  A list that grows as it is walked: ``modules()`` and ``parameters()``, which look
    for what comes twice, take three times as long, and a small step waits for the host."""
    found = list(modules)
    for m in found:
        found += [child for child in m._modules.values() if child is not None]  # noqa: SLF001
    return found


def _has_own_hook(module: nn.Module) -> bool:
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks  # noqa: SLF001
                or "forward" in module.__dict__)


def watched(module: nn.Module) -> bool:
    """Whether somebody gets to see what ``module`` itself takes and gives: a hook, its own or one of all modules, or a
    ``forward`` put in the place of its class's."""
    return bool(torch.nn.modules.module._has_any_global_hook()) or _has_own_hook(module)  # noqa: SLF001


def unobserved(*modules: nn.Module) -> bool:
    """Whether nobody looks into ``modules``: none in their trees is watched, by what would get to see the listed rows, moved
    together and with unwritten rows behind them, in the place of the batch's, and none is of a class of its own, which would
    run over those."""
    if torch.nn.modules.module._has_any_global_hook():  # noqa: SLF001
        return False
    return all(type(m) in _ROW_MODULES and not _has_own_hook(m) for m in _tree(modules))


@stops_at_count
class RMSNorm(nn.Module):
    def __init__(self, hidden_size: int, eps: float = 1e-6):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(hidden_size))
        self.variance_epsilon = eps

    def forward(self, x: torch.Tensor, live: torch.Tensor | None = None) -> torch.Tensor:
        return ops.rms_norm(x, self.weight, self.variance_epsilon, live=live)

    def fork(self, x: torch.Tensor, live: torch.Tensor | None = None) -> tuple[torch.Tensor, torch.Tensor]:
        """``(self(x), x)``: the input of a pre-norm block and its residual branch."""
        return ops.rms_norm_fork(x, self.weight, self.variance_epsilon, live=live)

    def extra_repr(self) -> str:
        return f"{tuple(self.weight.shape)}, eps={self.variance_epsilon}"


def norm_of_sum(norm: nn.Module, x: torch.Tensor, add: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """``(x + add, norm(x + add))``: a block's result, its residual added, and the next block's input; one launch for an ``RMSNorm``
    that nobody watches, any other module is called."""
    if type(norm) is RMSNorm and unobserved(norm):
        return ops.add_rms_norm(x, add, norm.weight, norm.variance_epsilon)
    x = x + add
    return x, norm(x)


def _init_linear_(weight: torch.Tensor, std: float = 0.02) -> None:
    with torch.no_grad():
        weight.normal_(mean=0.0, std=std)


@stops_at_count
class Linear(nn.Module):
    """Bias-optional linear layer; weight ``[out, in]`` like ``nn.Linear``."""

    def __init__(self, in_features: int, out_features: int, bias: bool = False, std: float = 0.02):
        super().__init__()
        self.in_features, self.out_features = in_features, out_features
        self.weight = nn.Parameter(torch.empty(out_features, in_features))
        self.bias = nn.Parameter(torch.zeros(out_features)) if bias else None
        # tensor parallelism (inference): ``row_parallel(x, weight, residual) -> sum over the ranks'
        # partial products + residual`` replaces the local product of a layer whose input is split
        self.row_parallel = None
        _init_linear_(self.weight, std)

    def forward(self, x: torch.Tensor, residual: torch.Tensor | None = None, live: torch.Tensor | None = None) -> torch.Tensor:
        if self.row_parallel is not None and self.bias is None:
            return self.row_parallel(x, self.weight, residual)
        return ops.linear(x, self.weight, self.bias, residual=residual, live=live)

    def extra_repr(self) -> str:
        return f"in={self.in_features}, out={self.out_features}, bias={self.bias is not None}"


@stops_at_count
class FusedLinear(nn.Module):
    """Several projections of the same input stored as one ``[sum(out), in]`` weight.

    ``names``/``sizes`` describe the parts.  ``state_dict`` exposes them as
    ``<prefix><name>.weight`` (and ``.bias``) exactly as separate ``nn.Linear``
    modules would, and loading accepts the split form, so checkpoints are
    indistinguishable from the unfused layout.
    """

    def __init__(self, in_features: int, names: list[str], sizes: list[int], bias: bool = False):
        super().__init__()
        self.in_features = in_features
        self.names, self.sizes = list(names), list(sizes)
        self.weight = nn.Parameter(torch.empty(sum(sizes), in_features))
        self.bias = nn.Parameter(torch.zeros(sum(sizes))) if bias else None
        _init_linear_(self.weight)
        self._register_state_dict_hook(FusedLinear._split_on_save)

    def attach(self, parent: nn.Module, attr: str) -> "FusedLinear":
        """Register the load-time merge on ``parent`` (the module that holds this
        layer as attribute ``attr``).  ``load_state_dict`` hands a child only the keys
        under the child's own prefix, so the split names ``<parent>.<part>.weight``
        are visible to the parent alone."""

        def merge(state_dict, prefix, *args):  # noqa: ANN001, ANN002
            for kind in ("weight", "bias"):
                keys = [f"{prefix}{name}.{kind}" for name in self.names]
                if all(k in state_dict for k in keys):
                    state_dict[f"{prefix}{attr}.{kind}"] = torch.cat([state_dict.pop(k) for k in keys], dim=0)

        parent._register_load_state_dict_pre_hook(merge)
        return self

    def offsets(self) -> list[int]:
        out, acc = [], 0
        for s in self.sizes:
            out.append(acc)
            acc += s
        return out

    def forward(self, x: torch.Tensor, live: torch.Tensor | None = None) -> torch.Tensor:
        return ops.linear(x, self.weight, self.bias, live=live)

    def forward_parts(self, x: torch.Tensor, first: int, last: int) -> torch.Tensor:
        """Apply only parts ``first .. last-1`` (row slice of the fused weight)."""
        offs = self.offsets() + [sum(self.sizes)]
        return ops.linear(x, self.weight, self.bias, rows=(offs[first], offs[last]))

    # the hooks see keys like "<prefix>weight"; the parent prefix (without this
    # module's own attribute name) is where the split names live.
    @staticmethod
    def _parent_prefix(prefix: str) -> str:
        trimmed = prefix[:-1] if prefix.endswith(".") else prefix
        return trimmed.rsplit(".", 1)[0] + "." if "." in trimmed else ""

    @staticmethod
    def _split_on_save(module, state_dict, prefix, local_metadata):  # noqa: ANN001, ARG004
        parent = FusedLinear._parent_prefix(prefix)
        for kind in ("weight", "bias"):
            fused = state_dict.pop(prefix + kind, None)
            if fused is None:
                continue
            for name, off, size in zip(module.names, module.offsets(), module.sizes):
                state_dict[f"{parent}{name}.{kind}"] = fused[off : off + size]
        return state_dict

    def extra_repr(self) -> str:
        parts = ", ".join(f"{n}:{s}" for n, s in zip(self.names, self.sizes))
        return f"in={self.in_features}, parts=[{parts}], bias={self.bias is not None}"


class RotaryTable(nn.Module):
    """fp32 cos/sin tables ``[max_pos, rot/2]`` (non-persistent buffers).

    Supports the ``default``, ``linear`` and ``llama3`` frequency schedules of
    Hugging Face ``rope_scaling`` / ``rope_parameters`` dicts.
    """

    def __init__(self, config: TransformerLayerConfig, max_positions: int | None = None):
        super().__init__()
        self.rot = config.rotary_dim
        self.head_dim = config.head_dim
        self.max_positions = int(max_positions or min(int(config.max_position_embeddings), 1 << 17))
        self.theta = float(config.rope_theta)
        scaling = config.get("rope_scaling") or config.get("rope_parameters") or {}
        if "sliding_attention" in scaling:
            scaling = scaling["sliding_attention"]
        self.scaling = dict(scaling) if isinstance(scaling, dict) else {}
        self.register_buffer("cos", torch.empty(0), persistent=False)
        self.register_buffer("sin", torch.empty(0), persistent=False)
        self._build(self.max_positions)

    def _inv_freq(self) -> torch.Tensor:
        rot = self.rot
        inv = 1.0 / (self.theta ** (torch.arange(0, rot, 2, dtype=torch.float64) / rot))
        kind = self.scaling.get("rope_type", self.scaling.get("type", "default"))
        if kind == "linear":
            inv = inv / float(self.scaling.get("factor", 1.0))
        elif kind == "llama3":
            factor = float(self.scaling.get("factor", 8.0))
            lo = float(self.scaling.get("low_freq_factor", 1.0))
            hi = float(self.scaling.get("high_freq_factor", 4.0))
            orig = float(self.scaling.get("original_max_position_embeddings", 8192))
            wavelen = 2 * math.pi / inv
            smooth = ((orig / wavelen) - lo) / (hi - lo)
            blended = (1 - smooth) * inv / factor + smooth * inv
            inv = torch.where(wavelen > orig / lo, inv / factor, torch.where(wavelen < orig / hi, inv, blended))
        return inv

    def _build(self, n: int) -> None:
        device = self.cos.device
        ang = torch.outer(torch.arange(n, dtype=torch.float64), self._inv_freq())
        self.cos = ang.cos().float().to(device).contiguous()
        self.sin = ang.sin().float().to(device).contiguous()
        self.max_positions = n

    def _apply(self, fn, recurse=True):  # noqa: ANN001
        """Keep the tables in fp32 whatever dtype the owning model is cast to."""
        super()._apply(fn, recurse)
        if self.cos.dtype != torch.float32:
            self.cos, self.sin = self.cos.float(), self.sin.float()
            self._build(self.max_positions)
        return self

    def ensure(self, max_pos: int) -> None:
        """Grow the tables (host side, outside any captured region) to cover ``max_pos``."""
        if max_pos >= self.max_positions:
            self._build(int(max_pos * 2))


@stops_at_count
class Attention(nn.Module):
    """Grouped-query self-attention over an ``AttnSpec`` mask.

    ``input_size`` differs from ``hidden_size`` only for the EAGLE-3 first layer,
    whose q/k/v projections read ``cat([embeds, hidden])`` (2H).
    """

    def __init__(self, config: TransformerLayerConfig, layer_idx: int, input_size: int | None = None, qk_norm: bool | None = None):
        super().__init__()
        self.layer_idx = layer_idx
        self.hidden_size = config.hidden_size
        self.nh, self.nkv, self.hd = config.num_attention_heads, config.num_key_value_heads, config.head_dim
        self.rot = config.rotary_dim
        self.scaling = self.hd**-0.5
        in_size = input_size or config.hidden_size
        self.qkv_proj = FusedLinear(
            in_size, ["q_proj", "k_proj", "v_proj"],
            [self.nh * self.hd, self.nkv * self.hd, self.nkv * self.hd], bias=bool(config.attention_bias),
        ).attach(self, "qkv_proj")
        self.o_proj = Linear(self.nh * self.hd, config.hidden_size, bias=bool(config.attention_bias))
        use_qk_norm = config.model_type.startswith("qwen3") if qk_norm is None else qk_norm
        self.q_norm = RMSNorm(self.hd, config.rms_norm_eps) if use_qk_norm else None
        self.k_norm = RMSNorm(self.hd, config.rms_norm_eps) if use_qk_norm else None

    def project_qkv(self, x: torch.Tensor, positions: torch.Tensor, rotary: RotaryTable, split: int | None = None, repeated: bool = False,
                    live: torch.Tensor | None = None):
        """x [T, in] -> (q [T, nh, hd], k [T, nkv, hd], v [T, nkv, hd]) with per-head
        norms (if any) and rotary embedding applied; with ``split`` k and v come as
        two tensors each, the rows below it and the rows from it on.  ``repeated``: ``x`` has
        ``split + 2`` rows, the rows from ``split`` on all read row ``split`` (``ops.repeat_rows``)."""
        T = positions.shape[0]
        nq, nk = self.nh * self.hd, self.nkv * self.hd
        qkv = self.qkv_proj(x, live)
        if self.q_norm is not None:
            return ops.norm_rope_heads(qkv, self.q_norm.weight, self.k_norm.weight, self.q_norm.variance_epsilon, positions, rotary.cos,
                                       rotary.sin, (self.nh, self.nkv, self.nkv), self.hd, self.rot, split, repeated, live)
        if repeated:
            qkv = ops.repeat_rows(qkv, T)
        q, k, v = ops.rope_split(qkv, positions, rotary.cos, rotary.sin, self.nh + self.nkv, self.hd, self.rot, nq, nk, live,
                                 unseen=not torch.is_grad_enabled() and unobserved(self.qkv_proj))
        q, k, v = q.view(T, self.nh, self.hd), k.view(T, self.nkv, self.hd), v.view(T, self.nkv, self.hd)
        return (q, k, v) if split is None else (q, k[:split], k[split:], v[:split], v[split:])

    def forward(self, x, positions, rotary, spec: AttnSpec, past: list | None = None, ctx_len: int | None = None,
                residual: torch.Tensor | None = None, repeated: bool = False, rows: ops.StepRows | None = None, dense: bool = False) -> torch.Tensor:
        """``past`` (EAGLE-3 TTT): list of (k, v) of earlier passes over the same
        positions.  Entry 0 is the context the interval part of ``spec`` indexes;
        later entries and this pass's own keys are reachable through
        ``spec.extra_idx`` (row ``(j-1)*T + i`` = key ``i`` of pass ``j``).

        ``ctx_len`` (P-EAGLE): the first ``ctx_len`` rows of this pass are the
        interval-addressed context, the remaining rows are the extra keys; ``repeated``
        says that ``x`` holds those only once (``project_qkv``).

        ``rows``: the rows that the step needs (``ops.step_rows``).  The inputs are of those rows, or of the whole batch
        (``dense``: keys and values of all rows are context), the result and ``spec`` are of those rows."""
        T = positions.shape[0]
        live = rows.live if rows is not None and not dense else None
        if ctx_len is not None and ctx_len < T:
            q, k_ctx, k_ext, v_ctx, v_ext = self.project_qkv(x, positions, rotary, split=ctx_len, repeated=repeated)
            out = ops.masked_attention(q, k_ctx, v_ctx, spec, k_ext, v_ext, scale=self.scaling)
            return self.o_proj(out.reshape(T, self.nh * self.hd), residual=residual)
        q, k, v = self.project_qkv(x, positions, rotary, live=live)
        if dense:
            live = rows.live
            q, residual = ops.take_rows(rows.index, rows.inverse, live, q.reshape(T, -1), residual)
            q = q.view(T, self.nh, self.hd)
        if past is None:
            out = ops.masked_attention(q, k, v, spec, scale=self.scaling)
        else:
            past.append((k, v))
            k_ctx, v_ctx = past[0]
            if len(past) > 1:
                k_ext, v_ext = past[1] if len(past) == 2 else (torch.cat([kv[i] for kv in past[1:]], dim=0) for i in range(2))
                out = ops.masked_attention(q, k_ctx, v_ctx, spec, k_ext, v_ext, scale=self.scaling)
            else:
                out = ops.masked_attention(q, k_ctx, v_ctx, spec, scale=self.scaling)
        return self.o_proj(out.reshape(T, self.nh * self.hd), residual=residual, live=live)


_GATE_ACTIVATIONS = {
    "gelu": lambda g: torch.nn.functional.gelu(g),
    "gelu_new": lambda g: torch.nn.functional.gelu(g, approximate="tanh"),
    "gelu_pytorch_tanh": lambda g: torch.nn.functional.gelu(g, approximate="tanh"),
    "relu": torch.relu,
}


@stops_at_count
class MLP(nn.Module):
    """Gated MLP ``down(act(gate(x)) * up(x))``.  SiLU (every supported verifier family's default)
    runs on the fused SwiGLU kernel; the other activations the reference accepts through
    ``--draft-hidden-act`` (GELU variants, ReLU) use the element-wise PyTorch formulation."""

    def __init__(self, config: TransformerLayerConfig, intermediate_size: int | None = None):
        super().__init__()
        inter = intermediate_size or config.intermediate_size
        self.hidden_act = str(config.hidden_act)
        if self.hidden_act not in ("silu", "swish") and self.hidden_act not in _GATE_ACTIVATIONS:
            raise ValueError(f"hidden_act={config.hidden_act!r} is not supported; choose one of {['silu', *sorted(_GATE_ACTIVATIONS)]}")
        self.gate_up_proj = FusedLinear(config.hidden_size, ["gate_proj", "up_proj"], [inter, inter], bias=bool(config.mlp_bias)).attach(self, "gate_up_proj")
        self.down_proj = Linear(inter, config.hidden_size, bias=bool(config.mlp_bias))

    def forward(self, x: torch.Tensor, residual: torch.Tensor | None = None, live: torch.Tensor | None = None) -> torch.Tensor:
        silu = self.hidden_act in ("silu", "swish")
        if silu and self.gate_up_proj.bias is None:
            hidden = ops.linear_swiglu(x, self.gate_up_proj.weight, live)  # activation in the GEMM's epilogue
            if hidden is not None:
                return self.down_proj(hidden, residual=residual, live=live)
        gate_up = self.gate_up_proj(x, live)
        if silu:
            hidden = ops.swiglu(gate_up, live)
        else:
            gate, up = gate_up.chunk(2, dim=-1)
            hidden = _GATE_ACTIVATIONS[self.hidden_act](gate) * up
        return self.down_proj(hidden, residual=residual, live=live)


# Rows x width from which on an EAGLE-3 or MTP step leaves out rows that nothing reads.  Listing them and copying queries and residuals costs
# four launches (20 us of a step); ms a step with all rows and with the needed ones, half of the rows supervised in spans of 64:
#   width 256:  513 rows 0.555 and 0.580, 1500 rows 0.723 and 0.731, 2048 rows 0.949 and 0.917, 4096 rows 1.200 and 1.129
#   width 1024: 257 rows 1.134 and 1.136, 513 rows 1.351 and 1.345, 1500 rows 2.051 and 1.873
#   width 4096: 257 rows 4.54 and 4.14, 800 rows 7.15 and 5.77, 1500 rows 10.77 and 8.14
# A batch that is supervised throughout pays for the listing and the copies: width 256, 2600 rows 1.097 and 1.124, 2048, 1001 rows 3.18 and
# 3.20, 4096, 2048 rows 14.06 and 14.07; multi-token prediction 4096, 2000 rows 21.9 and 22.0, with 256 experts 2048, 4096 rows 29.4 and 29.8.
NEEDED_ROWS_FROM = 1 << 19


def takes_listed_rows(layers, *linears: nn.Module) -> bool:
    """Whether decoder layers (``self_attn``, ``mlp``) and further linear layers may run over the rows that ``ops.step_rows``
    lists: every operator between them is a kernel that stops at the device's row count, nobody
    watches, and what is saved for the backward pass goes through no hook of the caller's, which would pack unwritten rows too."""
    if not unobserved(*layers) or torch._C._autograd._top_saved_tensors_default_hooks(True) is not None:  # noqa: SLF001
        return False
    linears = list(linears)
    for layer in layers:
        attn, mlp = layer.self_attn, layer.mlp
        if type(attn) is not Attention or type(mlp) is not MLP or mlp.hidden_act not in ("silu", "swish") or attn.hd not in (64, 128, 256) or attn.rot % 16:
            return False
        linears += [attn.qkv_proj, attn.o_proj, mlp.gate_up_proj, mlp.down_proj]
    return (
        ops.own_gemm_enabled()
        and all(p is None or p.is_cuda and p.dtype == torch.bfloat16 for m in _tree(layers) for p in m._parameters.values())  # noqa: SLF001
        and all(getattr(m, "bias", None) is None and getattr(m, "row_parallel", None) is None and m.weight.is_cuda and m.weight.dtype == torch.bfloat16
                and m.weight.is_contiguous() and m.weight.data_ptr() % 16 == 0 and m.weight.shape[0] % 8 == 0 and m.weight.shape[1] % 8 == 0
                and m.weight.shape[1] <= 1 << 20 for m in linears)
    )


@stops_at_count
class DecoderLayer(nn.Module):
    """Pre-norm decoder block (Llama / Qwen3 layout)."""

    def __init__(self, config: TransformerLayerConfig, layer_idx: int):
        super().__init__()
        self.self_attn = Attention(config, layer_idx)
        self.mlp = MLP(config)
        self.input_layernorm = RMSNorm(config.hidden_size, config.rms_norm_eps)
        self.post_attention_layernorm = RMSNorm(config.hidden_size, config.rms_norm_eps)

    def forward(self, x, positions, rotary, spec, past=None, ctx_len=None, rows=None, dense=False) -> torch.Tensor:
        """``rows``, ``dense``: as in ``Attention``."""
        live = rows.live if rows is not None else None
        normed, x = self.input_layernorm.fork(x, None if dense else live)
        x = self.self_attn(normed, positions, rotary, spec, past, ctx_len, residual=x, rows=rows, dense=dense)
        normed, x = self.post_attention_layernorm.fork(x, live)
        return self.mlp(normed, residual=x, live=live)


def _of_one_call(layer: nn.Module, next_norm: nn.Module | None) -> bool:
    """Whether ``decoder_layer_fwd`` does what calling the modules does: every one of the class whose formula it has (other norms
    have a ``weight`` and an epsilon, too), none watched, no bias, no exchange between ranks."""
    if type(layer) is not DecoderLayer or not unobserved(layer) or (next_norm is not None and not unobserved(next_norm)):
        return False
    attn, mlp = layer.self_attn, layer.mlp
    if type(attn) is not Attention or type(mlp) is not MLP or mlp.hidden_act not in ("silu", "swish"):
        return False
    heads = [attn.q_norm, attn.k_norm] if attn.q_norm is not None or attn.k_norm is not None else []
    norms = [layer.input_layernorm, layer.post_attention_layernorm, *heads, *([] if next_norm is None else [next_norm])]
    return (all(type(n) is RMSNorm for n in norms)
            and all(type(m) is FusedLinear and m.bias is None for m in (attn.qkv_proj, mlp.gate_up_proj))
            and all(type(m) is Linear and m.bias is None and m.row_parallel is None for m in (attn.o_proj, mlp.down_proj)))


def decoder_layer_fwd(layer: DecoderLayer, h: torch.Tensor, normed: torch.Tensor | None, next_norm: RMSNorm | None, positions, rotary: RotaryTable, spec):
    """A decoder layer's result without a gradient, in one call of the extension: ``(h, next_norm(h) or None)``, or ``None`` where
    its modules have to be called (other devices, types or activations, biases, a watched module).  ``normed``: the layer's input
    behind its first norm, if the layer before has formed it.  The launches are those of the modules."""
    from speculators_b200.ops import attention_cuda

    if (not h.is_cuda or h.dtype != torch.bfloat16 or torch.is_grad_enabled() or torch.autograd.forward_ad._current_level >= 0
            or spec.extra_idx is not None or not ops.own_gemm_enabled() or not ops.fused_swiglu_enabled() or attention_cuda.FWD_IMPL != "tc"
            or not _of_one_call(layer, next_norm)):
        return None
    attn, mlp = layer.self_attn, layer.mlp
    qkv, o, gate_up, down = attn.qkv_proj, attn.o_proj, mlp.gate_up_proj, mlp.down_proj
    q_norm, k_norm = attn.q_norm, attn.k_norm
    first, post = layer.input_layernorm, layer.post_attention_layernorm
    out = ops.native().decoder_layer_fwd(
        h, normed, first.weight, qkv.weight, None if q_norm is None else q_norm.weight, None if k_norm is None else k_norm.weight, o.weight, post.weight,
        gate_up.weight, down.weight, None if next_norm is None else next_norm.weight, positions, rotary.cos, rotary.sin, spec.lo, spec.hi, attn.nh, attn.nkv,
        attn.hd, attn.rot, first.variance_epsilon, 0.0 if q_norm is None else q_norm.variance_epsilon, post.variance_epsilon,
        0.0 if next_norm is None else next_norm.variance_epsilon, attn.scaling, attention_cuda.tensor_core_shape(h.shape[0], attn.hd, None), ops.gemm_status(h.device))
    if not out:
        return None
    return out[0], out[1] if next_norm is not None else None
