"""EAGLE-3 steps over the rows that a loss term or counter reads: the plan, the kernels that stop at a device-side row count,
and the whole pass against the pass over all rows."""

import copy
import warnings

import pytest
import torch

from conftest import make_tiny_batch, make_tiny_eagle3

import speculators_b200 as sb
from speculators_b200 import ops
from speculators_b200.layer_config import TransformerLayerConfig
from speculators_b200.models.eagle3 import Eagle3DraftModel, Eagle3SpeculatorConfig
from speculators_b200.models.eagle3.attention import causal_document_interval


def _mask(kind: str, T: int, device="cpu") -> torch.Tensor:
    g = torch.Generator().manual_seed(T)
    m = torch.zeros(T, dtype=torch.bool)
    if kind == "spans":
        m = (torch.rand((T + 31) // 32, generator=g) < 0.5).repeat_interleave(32)[:T]
    elif kind == "scattered":
        m = torch.rand(T, generator=g) < 0.2
    elif kind == "all":
        m[:] = True
    elif kind == "ends":
        m[0] = m[-1] = True
    return m.to(device)


KINDS = ["spans", "scattered", "all", "none", "ends"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("layers", [1, 2])
def test_pass_over_needed_rows_equals_the_whole_pass(tiny_verifier_dir, tiny_vocab_maps, monkeypatch, kind, layers):
    model = make_tiny_eagle3(tiny_verifier_dir, tiny_vocab_maps, num_layers=layers)
    kwargs, _ = sb.Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
    batch = make_tiny_batch()
    batch["loss_mask"] = _mask(kind, batch["loss_mask"].shape[1])[None]
    results = []
    for needed in (False, True):
        monkeypatch.setattr(Eagle3DraftModel, "_takes_needed_rows", lambda *_, n=needed: n)
        model.zero_grad()
        _, loss, metrics = model(**batch, **kwargs)
        loss.backward()
        results.append((metrics, {n: p.grad.clone() for n, p in model.named_parameters() if p.grad is not None}))
    (metrics, grads), (metrics_needed, grads_needed) = results
    assert metrics.keys() == metrics_needed.keys() and grads.keys() == grads_needed.keys()
    for k, v in metrics.items():
        torch.testing.assert_close(metrics_needed[k], v, rtol=1e-5, atol=1e-6, msg=k)
    for n, v in grads.items():
        torch.testing.assert_close(grads_needed[n], v, rtol=1e-4, atol=1e-5 * float(v.abs().max()) + 1e-9, msg=n)


# --------------------------------------------------------------------------- on a GPU
def _poison():
    """What is allocated from here on and not written holds NaN: free memory does, and nothing freed earlier is left beside it."""
    torch.cuda.empty_cache()
    held = [torch.full((1 << 27,), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    del held


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 255, 256, 257, 1000, 1024, 8192, 8200, 20011])
@pytest.mark.parametrize("kind", KINDS)
def test_plan(T, kind):
    S = 3
    g = torch.Generator().manual_seed(0)
    doc = torch.arange(T) // 300
    doc[T - T // 50 :] = -1
    mask, ids, pos = _mask(kind, T), torch.randint(0, 1000, (T,), generator=g), torch.arange(T) % 300
    iv = causal_document_interval(doc, 64)
    full = causal_document_interval(doc, None)
    ref = ops.step_rows(mask, ids, pos, [iv, full], S)
    got = ops.step_rows(mask.cuda(), ids.cuda(), pos.cuda(), [tuple(t.cuda() for t in iv), causal_document_interval(doc.cuda(), None)], S)
    for index, live, ref_index, ref_live in ((got.index, got.live, ref.index, ref.live), (got.target_index, got.target_live, ref.target_index, ref.target_live)):
        n, want = int(live), int(ref_live)
        assert n == min(T, max(256, -(-want // 256) * 256))
        rows = index[:n].cpu()
        assert (rows[1:] > rows[:-1]).all() and set(ref_index[:want].tolist()) <= set(rows.tolist())
    n = int(got.live)
    rows = got.index[:n].cpu()
    inverse = torch.full((T,), -1, dtype=torch.int32)
    inverse[rows] = torch.arange(n, dtype=torch.int32)
    assert torch.equal(got.inverse.cpu(), inverse)
    target_rows = got.target_index[: int(got.target_live)].cpu()
    target_inverse = torch.full((T + S,), -1, dtype=torch.int32)
    target_inverse[target_rows] = torch.arange(len(target_rows), dtype=torch.int32)
    assert torch.equal(got.prev_correct.cpu(), torch.cat([mask[rows], torch.zeros(T - n, dtype=torch.bool)]))
    for (lo, hi), (want_lo, want_hi) in zip(got.intervals, (iv, full)):
        assert torch.equal(lo[:n].cpu(), want_lo[rows]) and torch.equal(hi[:n].cpu(), want_hi[rows]) and not lo[n:].any() and not hi[n:].any()
    padded_mask, padded_ids = torch.cat([mask, mask.new_zeros(S)]), torch.cat([ids, ids.new_zeros(S)])
    for s in range(S):
        assert torch.equal(got.ids[s, :n].cpu(), padded_ids[rows + s]) and not got.ids[s, n:].any()
        assert torch.equal(got.positions[s, :n].cpu(), pos[rows] + s)
        assert torch.equal(got.mask[s, :n].cpu(), padded_mask[rows + s]) and not got.mask[s, n:].any()
        assert torch.equal(got.target_row[s, :n].cpu(), target_inverse[rows + s]) and (got.target_row[s, n:] == -1).all()
        wanted = padded_mask[rows + s] | mask[rows] & (rows + s < T)
        assert (got.target_row[s, :n].cpu()[wanted] >= 0).all()
        if s:
            want = torch.arange(s)[None, :] * T + torch.arange(n)[:, None]
            assert torch.equal(got.extra[s][:n].cpu().long(), want) and (got.extra[s][n:] == -1).all()


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 3, 4, 5, 10, 11, 12, 13])
@pytest.mark.parametrize("live", [256, 768, 1001])
def test_products_stop_at_the_count(variant, live):
    """Rows behind hold NaN: neither read (weight gradient, which sums over them) nor written."""
    T, M, N = 1001, 384, 1032
    g = torch.Generator(device="cuda").manual_seed(variant * 7 + live)
    a = torch.randn(T, M, generator=g, device="cuda").bfloat16()
    w = torch.randn(N, M, generator=g, device="cuda").bfloat16()
    dy = torch.randn(T, N, generator=g, device="cuda").bfloat16()
    a[live:], dy[live:] = float("nan"), float("nan")
    count, status = torch.tensor([live], dtype=torch.int32, device="cuda"), ops.gemm_status(a.device)
    res = torch.randn(T, N, generator=g, device="cuda").bfloat16()
    out, summed, dx = (torch.full((T, k), 7.0, dtype=torch.bfloat16, device="cuda") for k in (N, N, M))
    dw = torch.full((N, M), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.native().gemm_tn_variant(a, w, out, None, 0, status, variant, count)
    ops.native().gemm_tn_variant(a, w, summed, res, 2, status, variant, count)
    ops.native().gemm_variant(dy, w, dx, 0, False, True, status, variant, count)
    ops.native().gemm_variant(dy, a, dw, 0, True, True, status, variant, count)
    af, wf, df = a[:live].float(), w.float(), dy[:live].float()
    for got, want in ((out[:live], af @ wf.T), (summed[:live], af @ wf.T + res[:live].float()), (dx[:live], df @ wf), (dw, df.T @ af)):
        assert float((got.float() - want).norm() / want.norm()) < 4e-3  # one rounding to bf16 (2^-9 at most, relative)
    for t in (out, summed, dx):
        assert (t[live:] == 7.0).all()
    assert int(status) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("lives", [(256, 512, None), (None, 256, 768), (1001, 1001, 256)])
def test_weight_gradient_parts_stop_at_their_counts(lives):
    T, M, N = 1001, 2560, 2048
    g = torch.Generator(device="cuda").manual_seed(1)
    dys, xs, counts, want = [], [], [], 0
    for live in lives:
        dy, x = (torch.randn(T, k, generator=g, device="cuda").bfloat16() for k in (M, N))
        n = T if live is None else live
        dy[n:], x[n:] = float("nan"), float("nan")
        want = want + dy[:n].float().T @ x[:n].float()
        dys.append(dy), xs.append(x)
        counts.append(torch.empty(0, dtype=torch.int32, device="cuda") if live is None else torch.tensor([live], dtype=torch.int32, device="cuda"))
    dw = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    status = ops.gemm_status(dw.device)
    ops.native().gemm_wgrad_parts_rows(dys, xs, dw, False, status, counts)
    assert float((dw.float() - want).norm() / want.norm()) < 4e-3 and int(status) == 0


def _model(layers, head_dim, qwen, inter, window):
    cfg = dict(architectures=["Qwen3ForCausalLM" if qwen else "LlamaForCausalLM"], model_type="qwen3" if qwen else "llama", hidden_size=256, num_hidden_layers=layers,
               num_attention_heads=4, num_key_value_heads=2, head_dim=head_dim, intermediate_size=inter, vocab_size=1024, rms_norm_eps=1e-5, rope_theta=10000.0,
               max_position_embeddings=4096, hidden_act="silu")
    if window:
        cfg.update(sliding_window=200, layer_types=["sliding_attention"] + ["full_attention"] * (layers - 1))
    torch.manual_seed(0)
    model = Eagle3DraftModel(Eagle3SpeculatorConfig(transformer_layer_config=TransformerLayerConfig(**cfg), draft_vocab_size=512, norm_before_residual=bool(window),
                                                    norm_before_fc=True, norm_output=qwen, eagle_aux_hidden_state_layer_ids=[2, 5, 8]))
    model.load_verifier_weights()
    with torch.no_grad():
        model.embed_tokens.weight.normal_(0.0, 1.0)
        model.lm_head.weight.normal_(0.0, 0.1)
        model.verifier_lm_head.weight.copy_(model.lm_head.weight)
    kept = torch.arange(512) * 2
    t2d = torch.zeros(1024, dtype=torch.bool)
    t2d[kept] = True
    model.load_vocab_mappings(t2d, kept - torch.arange(512))
    return model.cuda().bfloat16()


def _gpu_batch(T, kind):
    g = torch.Generator().manual_seed(T)
    doc = torch.arange(T) // max(1, T // 3)
    doc[T - 17 :] = -1
    mask = _mask(kind, T)
    mask[T - 17 :] = False
    return {"input_ids": torch.randint(0, 1024, (1, T), generator=g).cuda(), "hidden_states": torch.randn(1, T, 768, generator=g).bfloat16().cuda(),
            "verifier_last_hidden_states": torch.randn(1, T, 256, generator=g).bfloat16().cuda(), "document_ids": doc[None].cuda(),
            "loss_mask": mask[None].cuda(), "position_ids": (torch.arange(T) % 400)[None].cuda()}


@pytest.mark.gpu
@pytest.mark.parametrize("T", [513, 777, 1536])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("layers,head_dim,qwen,inter,window", [(1, 64, False, 688, True), (1, 128, True, 512, True), (2, 128, False, 512, False), (1, 256, True, 512, False)])
def test_gpu_pass_over_needed_rows(monkeypatch, T, kind, layers, head_dim, qwen, inter, window):
    model, batch = _model(layers, head_dim, qwen, inter, window), _gpu_batch(T, kind)
    kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
    results = []
    for needed in (False, True):
        monkeypatch.setattr(Eagle3DraftModel, "_takes_needed_rows", lambda *_, n=needed: n)
        for p in model.parameters():
            p.grad = None
        _poison()
        _, loss, metrics = model(**batch, **kwargs)
        loss.backward()
        results.append(({k: v.float().cpu() for k, v in metrics.items()}, {n: p.grad.float() for n, p in model.named_parameters() if p.grad is not None}))
    (metrics, grads), (metrics_needed, grads_needed) = results
    assert metrics.keys() == metrics_needed.keys() and grads.keys() == grads_needed.keys()
    for k, v in metrics.items():  # the same bits per row; fp32 sums in another order
        torch.testing.assert_close(metrics_needed[k], v, rtol=2e-4, atol=1e-6, msg=k)
    for n, v in grads.items():
        # gradients round to bf16 (2^-9) on the way and at the end; sums over rows and queries take another order in between
        assert torch.isfinite(grads_needed[n]).all(), n
        assert float((grads_needed[n] - v).norm()) <= 1e-2 * float(v.norm()) + 1e-12, (n, float((grads_needed[n] - v).norm() / v.norm()))
    ops.check_gemm_status()


@pytest.mark.gpu
def test_gpu_what_is_not_one_fused_loss_takes_all_rows():
    model, batch = _model(1, 64, False, 512, False), _gpu_batch(2100, "spans")
    for loss_fn, implementation, want in (("kl_div", "fused", True), ("ce", "fused", True), ("kl_div", "eager", False), ('{"ce": 0.5, "tv": 0.5}', "fused", False), ("nla", "fused", False)):
        kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn=loss_fn, loss_implementation=implementation, ttt_steps=2, ttt_step_loss_decay=1.0)
        assert model._takes_needed_rows(2100, batch["loss_mask"], kwargs["loss_config"], 2) is want, loss_fn
    assert not model._takes_needed_rows(2100, None, None, 2) and not model._takes_needed_rows(2047, batch["loss_mask"][:, :2047], None, 2)
    tokens, loss, _ = model(**batch, ttt_steps=2)  # draft tokens of every row
    assert len(tokens) == 2 and tokens[0].shape == (1, 2100)
    assert not copy.deepcopy(model).float()._takes_needed_rows(2100, batch["loss_mask"], None, 2)


# --------------------------------------------------------------------------- multi-token prediction
def _mtp(experts: int, hidden: int, head_dim: int, vocab: int):
    from speculators_b200.config import SpeculatorsConfig, VerifierConfig
    from speculators_b200.models.mtp import MTPDraftModel, MTPSpeculatorConfig
    from speculators_b200.proposals.greedy import GreedyTokenProposalConfig

    cfg = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=hidden, num_hidden_layers=4, num_attention_heads=4, num_key_value_heads=2,
               head_dim=head_dim, intermediate_size=2 * hidden, vocab_size=vocab, rms_norm_eps=1e-6, rope_theta=10000.0, max_position_embeddings=4096,
               hidden_act="silu")
    if experts:
        cfg.update(architectures=["Qwen3NextForCausalLM"], model_type="qwen3_next", partial_rotary_factor=0.25, num_experts=experts, num_experts_per_tok=2,
                   moe_intermediate_size=256, shared_expert_intermediate_size=256, norm_topk_prob=True, decoder_sparse_step=1, mlp_only_layers=[])
    torch.manual_seed(0)
    model = MTPDraftModel(MTPSpeculatorConfig(transformer_layer_config=TransformerLayerConfig(**cfg), speculators_config=SpeculatorsConfig(
        algorithm="mtp", proposal_methods=[GreedyTokenProposalConfig(speculative_tokens=3)], default_proposal_method="greedy",
        verifier=VerifierConfig(name_or_path=None, architectures=cfg["architectures"]))))
    model.load_verifier_weights()
    with torch.no_grad():
        model.embed_tokens.weight.normal_(0.0, 1.0)
        model.lm_head.weight.normal_(0.0, 0.1)
    model.embed_tokens.weight.requires_grad_(False)
    model.lm_head.weight.requires_grad_(False)
    return model


def _mtp_results(model, batch, monkeypatch):
    results = []
    for needed in (False, True):
        monkeypatch.setattr(type(model), "_takes_needed_rows", lambda *_, n=needed: n)
        for p in model.parameters():
            p.grad = None
        if batch["input_ids"].is_cuda:
            _poison()
        logits, loss, metrics = model(**batch, return_logits=False, step_weights=[0.5, 0.3, 0.2])
        assert logits == []
        loss.backward()
        results.append((metrics, {n: p.grad.float() for n, p in model.named_parameters() if p.grad is not None}))
    return results


@pytest.mark.parametrize("kind", KINDS)
def test_mtp_step_over_needed_rows_equals_the_whole_step(monkeypatch, kind):
    T, model = 50, _mtp(0, 32, 8, 64)
    batch = {"input_ids": torch.randint(0, 64, (1, T)), "hidden_states": torch.randn(1, T, 32), "loss_mask": _mask(kind, T)[None]}
    monkeypatch.setattr(type(model.mtp_layers[0]), "takes_listed_rows", lambda _: True)
    (metrics, grads), (metrics_needed, grads_needed) = _mtp_results(model, batch, monkeypatch)
    assert metrics.keys() == metrics_needed.keys() and grads.keys() == grads_needed.keys()
    for k, v in metrics.items():
        torch.testing.assert_close(metrics_needed[k], v, rtol=1e-5, atol=1e-6, msg=k)
    for n, v in grads.items():
        torch.testing.assert_close(grads_needed[n], v, rtol=1e-4, atol=1e-5 * float(v.abs().max()) + 1e-9, msg=n)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [516, 777, 1540])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("experts,head_dim", [(0, 128), (0, 64), (8, 256)])
def test_gpu_mtp_step_over_needed_rows(monkeypatch, T, kind, experts, head_dim):
    g = torch.Generator().manual_seed(T)
    model = _mtp(experts, 512, head_dim, 1000).cuda().bfloat16()
    assert model.mtp_layers[0].takes_listed_rows()
    batch = {"input_ids": torch.randint(0, 1000, (1, T), generator=g).cuda(), "hidden_states": torch.randn(1, T, 512, generator=g).bfloat16().cuda(),
             "loss_mask": _mask(kind, T)[None].cuda()}
    (metrics, grads), (metrics_needed, grads_needed) = _mtp_results(model, batch, monkeypatch)
    assert metrics.keys() == metrics_needed.keys() and grads.keys() == grads_needed.keys()
    for k, v in metrics.items():
        torch.testing.assert_close(metrics_needed[k], v, rtol=2e-4, atol=1e-6, msg=k)
    for n, v in grads.items():  # as for EAGLE-3
        assert torch.isfinite(grads_needed[n]).all(), n
        assert float((grads_needed[n] - v).norm()) <= 1e-2 * float(v.norm()) + 1e-12, (n, float((grads_needed[n] - v).norm() / v.norm()))
    ops.check_gemm_status()


# --------------------------------------------------------------------------- who watches sees the whole batch
def _watched(model, where, seen):
    """A hook, of one kind or another, that keeps what the module at ``where`` takes or gives."""
    place, _, kind = where.partition(":")
    module = {"layer": lambda: model.layers[0], "mlp": lambda: model.layers[0].mlp, "norm": lambda: model.norm, "verifier_norm": lambda: model.verifier_norm,
              "embed_tokens": lambda: model.embed_tokens}[place]()

    def keep(tensors):
        seen.append([t.detach().clone() for t in (tensors if isinstance(tensors, tuple) else (tensors,)) if isinstance(t, torch.Tensor)])

    if kind == "pre":
        return module.register_forward_pre_hook(lambda m, args: keep(args))
    if kind == "backward":
        return module.register_full_backward_hook(lambda m, taken, given: keep(given))
    if kind == "global":
        return torch.nn.modules.module.register_module_forward_hook(lambda m, args, out: keep(out) if m is module else None)
    return module.register_forward_hook(lambda m, args, out: keep(out))


@pytest.mark.parametrize("register", ["register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook", "register_full_backward_pre_hook"])
def test_hooks_are_noticed(register):
    from speculators_b200.models.layers import unobserved

    layer = _mtp(0, 32, 8, 64).mtp_layers[0]
    for module in (layer, layer.mlp.down_proj):
        handle = getattr(module, register)(lambda *_: None)
        assert not unobserved(layer) and not unobserved(torch.nn.Identity(), layer)
        handle.remove()
        assert unobserved(layer)
    handle = torch.nn.modules.module.register_module_forward_pre_hook(lambda *_: None)
    assert not unobserved(layer)
    handle.remove()
    assert unobserved(layer)


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["layer", "layer:pre", "layer:backward", "mlp", "mlp:global", "norm", "verifier_norm", "embed_tokens"])
def test_gpu_hooks_see_the_rows_of_the_batch(monkeypatch, where):
    model, batch = _model(1, 64, False, 688, True), _gpu_batch(2100, "spans")
    kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
    results = []
    for whole in (True, False):
        with monkeypatch.context() as patched:
            if whole:
                patched.setattr(Eagle3DraftModel, "_takes_needed_rows", lambda *_: False)
            seen = []
            handle = _watched(model, where, seen)
            _poison()
            _, loss, _ = model(**batch, **kwargs)
            loss.backward()
            handle.remove()
            results.append(seen)
    want, got = results
    assert len(got) == len(want) == (1 if where == "verifier_norm" else 3)
    for a, b in zip(got, want):
        assert len(a) == len(b) > 0
        for x, y in zip(a, b):  # the same route: the same bits but for the atomics behind the gradients of irregular extra keys
            assert x.shape == y.shape and float((x.float() - y.float()).norm()) <= 1e-2 * float(y.float().norm())
    assert model._takes_needed_rows(2100, batch["loss_mask"], kwargs["loss_config"], 3)  # and nobody watches any more


@pytest.mark.gpu
@pytest.mark.parametrize("experts", [0, 8])
def test_gpu_mtp_hooks_see_the_rows_of_the_batch(experts):
    T = 1540
    model = _mtp(experts, 512, 256 if experts else 64, 1000).cuda().bfloat16()
    batch = {"input_ids": torch.randint(0, 1000, (1, T)).cuda(), "hidden_states": torch.randn(1, T, 512).bfloat16().cuda(), "loss_mask": _mask("spans", T)[None].cuda()}
    results = []
    for kwargs in ({"return_logits": True}, {"return_logits": False}):
        seen = []
        with torch.no_grad():
            handle = model.mtp_layers[0].register_forward_hook(lambda m, args, out: seen.append(out.clone()))
            _poison()
            model(**batch, **kwargs)
            handle.remove()
        results.append(seen)
    want, got = results
    assert len(want) == len(got) == 3
    for a, b in zip(got, want):
        assert torch.equal(a, b)




class _WithAdapter(torch.nn.Module):
    """What ``_adapted`` puts behind a linear layer: a trained path over every row that comes in."""

    def __init__(self, width_in: int, width_out: int):
        super().__init__()
        self.a, self.b = torch.nn.Parameter(torch.randn(8, width_in) * 0.05), torch.nn.Parameter(torch.randn(width_out, 8) * 0.05)

    def forward(self, x):
        return x @ self.a.T @ self.b.T


def _adapted(linear, as_class: bool):
    linear.adapter = _WithAdapter(linear.in_features, linear.out_features).to(linear.weight.device, linear.weight.dtype)
    base = type(linear).forward
    if as_class:
        class Adapted(type(linear)):
            def forward(self, x, residual=None, live=None):
                return base(self, x, residual=residual, live=live) + self.adapter(x)

        linear.__class__ = Adapted
    else:
        linear.forward = lambda x, residual=None, live=None: base(linear, x, residual=residual, live=live) + linear.adapter(x)


def test_modules_of_the_users_own_are_noticed():
    from speculators_b200.models.layers import RMSNorm, unobserved

    class Own(RMSNorm):
        pass

    for experts in (0, 8):
        layer = _mtp(experts, 512, 256, 64).mtp_layers[0]
        assert unobserved(layer)
        norm = layer.final_layernorm
        layer.final_layernorm = Own(512)
        assert not unobserved(layer)
        layer.final_layernorm = norm
        assert unobserved(layer)
        norm.forward = lambda x, live=None: x
        assert not unobserved(layer)


@pytest.mark.gpu
def test_gpu_a_verifier_norm_of_the_users_own_is_called(monkeypatch):
    """Whatever it has for weights."""
    model, batch = _model(1, 64, False, 688, True), _gpu_batch(2100, "spans")
    kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)

    class Halved(type(model.verifier_norm)):
        def forward(self, x):
            return super().forward(x) * 0.5

    halved = Halved(256).cuda().bfloat16()
    for norm in (halved, torch.nn.Identity()):
        model.verifier_norm = norm
        losses = []
        for whole in (True, False):
            with monkeypatch.context() as patched, torch.no_grad():
                if whole:
                    patched.setattr(Eagle3DraftModel, "_takes_needed_rows", lambda *_: False)
                losses.append(float(model(**batch, **kwargs)[1]))
        assert losses[0] == losses[1]


@pytest.mark.gpu
@pytest.mark.parametrize("as_class", [True, False])
@pytest.mark.parametrize("algorithm", ["eagle3", "mtp"])
def test_gpu_modules_of_the_users_own_run_over_the_rows_of_the_batch(monkeypatch, algorithm, as_class):
    torch.manual_seed(3)
    if algorithm == "eagle3":
        model, batch = _model(1, 64, False, 688, True), _gpu_batch(2100, "spans")
        kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
    else:
        model = _mtp(0, 512, 64, 1000).cuda().bfloat16()
        batch = {"input_ids": torch.randint(0, 1000, (1, 1540)).cuda(), "hidden_states": torch.randn(1, 1540, 512).bfloat16().cuda(), "loss_mask": _mask("spans", 1540)[None].cuda()}
        kwargs = {"return_logits": False}
    _adapted(model.layers[0].mlp.down_proj, as_class)
    results = []
    for whole in (True, False):
        with monkeypatch.context() as patched:
            if whole:
                patched.setattr(type(model), "_takes_needed_rows", lambda *_: False)
            for p in model.parameters():
                p.grad = None
            _poison()
            _, loss, _ = model(**batch, **kwargs)
            loss.backward()
            results.append([float(loss)] + [p.grad.float() for p in model.layers[0].mlp.down_proj.adapter.parameters()])
    (loss, *grads), (loss_got, *grads_got) = results
    assert abs(loss_got - loss) <= 2e-4 * abs(loss)
    for got, want in zip(grads_got, grads):  # rounded to bf16 on the way, sums in another order (MTP's head takes the listed rows)
        assert float((got - want).norm()) <= 1e-2 * float(want.norm())


def test_trainer_asks_for_logits_that_somebody_takes():
    from types import SimpleNamespace

    from speculators_b200.models.mtp import MTPDraftModel
    from speculators_b200.train import Trainer

    class Reads(MTPDraftModel):
        def forward(self, *args, **kwargs):
            logits, loss, metrics = super().forward(*args, **kwargs)
            metrics["peak"] = logits[0].max()
            return logits, loss, metrics

    class Keeps(MTPDraftModel):
        pass

    def asked(model):
        return Trainer.loss_only(SimpleNamespace(model=model), {"step_weights": None})

    def of(cls):
        model = _mtp(0, 32, 8, 64)
        model.__class__ = cls
        return model

    lean, full = {"return_logits": False, "step_weights": None}, {"step_weights": None}
    assert asked(of(MTPDraftModel)) == lean and asked(of(Keeps)) == lean
    assert asked(of(Reads)) == full
    model = of(MTPDraftModel)
    handle = model.register_forward_hook(lambda m, args, out: None)
    assert asked(model) == full
    handle.remove()
    assert asked(model) == lean
    model.forward = lambda *args, **kwargs: MTPDraftModel.forward(model, *args, **kwargs)
    assert asked(model) == full
    assert asked(torch.nn.Identity()) == full


@pytest.mark.gpu
@pytest.mark.parametrize("algorithm", ["eagle3", "eagle3 head norms", "mtp", "mtp experts"])
@pytest.mark.parametrize("forward_too", [True, False])
def test_gpu_anomaly_detection_finds_nothing_in_a_sound_step(monkeypatch, algorithm, forward_too):
    """It looks for NaN in every gradient, also in rows that nobody wrote."""
    if algorithm.startswith("eagle3"):
        qwen = algorithm.endswith("norms")
        model, batch = _model(2 if qwen else 1, 64, qwen, 688, True), _gpu_batch(2100, "spans")
        kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
    else:
        experts = 8 if algorithm.endswith("experts") else 0
        model = _mtp(experts, 512, 256 if experts else 64, 1000).cuda().bfloat16()
        batch = {"input_ids": torch.randint(0, 1000, (1, 1540)).cuda(), "hidden_states": torch.randn(1, 1540, 512).bfloat16().cuda(), "loss_mask": _mask("spans", 1540)[None].cuda()}
        kwargs = {"return_logits": False}
    taken = []
    monkeypatch.setattr(ops, "step_rows", lambda *args, made=ops.step_rows, **kw: taken.append(1) or made(*args, **kw))
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")  # that it is slow
        with torch.autograd.set_detect_anomaly(forward_too):
            _poison()
            _, loss, _ = model(**batch, **kwargs)
        _poison()
        with torch.autograd.set_detect_anomaly(True):
            loss.backward()
    assert taken and torch.isfinite(loss)
    assert all(torch.isfinite(p.grad).all() for p in model.parameters() if p.grad is not None)


# --------------------------------------------------------------------------- one graph, batches of any density
@pytest.mark.gpu
@pytest.mark.parametrize("algorithm", ["eagle3", "mtp", "mtp experts"])
def test_gpu_one_graph_replayed_over_masks_of_any_density(monkeypatch, tmp_path, algorithm):
    """The rows are listed inside the graph: a replay with fewer or more of them than the capture had gives that batch's gradients."""
    from speculators_b200.train import Trainer, TrainerConfig
    from speculators_b200.train.synthetic import SyntheticLoader

    if algorithm == "eagle3":
        model, batch = _model(1, 64, False, 688, True), _gpu_batch(2100, "all")
        kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
        T, cls = 2100, Eagle3DraftModel
        lossy = batch["loss_mask"].clone()
    else:
        experts = 8 if algorithm.endswith("experts") else 0
        T, model = 1540, _mtp(experts, 512, 256 if experts else 64, 1000).cuda().bfloat16()
        g = torch.Generator().manual_seed(1)
        batch = {"input_ids": torch.randint(0, 1000, (1, T), generator=g).cuda(), "hidden_states": torch.randn(1, T, 512, generator=g).bfloat16().cuda()}
        lossy, kwargs, cls = torch.ones(1, T, dtype=torch.bool, device="cuda"), {"step_weights": [0.5, 0.3, 0.2]}, type(model)
    g = torch.Generator().manual_seed(5)
    at = torch.rand((T + 31) // 32, generator=g).repeat_interleave(32)[:T].cuda()[None]

    def trainer(graph):
        return Trainer(copy.deepcopy(model), TrainerConfig(lr=0.0, weight_decay=0.0, num_epochs=1, save_path=str(tmp_path), train_call_kwargs=kwargs, scheduler_type="none",
                                                           log_freq=10**9, use_cuda_graph=graph, device="cuda:0"), SyntheticLoader([batch], 1))

    graphed, eager = trainer(True), trainer(False)
    for density in (0.6, 0.0, 1.0, 0.2, 0.6, 0.0, 0.2, 1.0):
        one = dict(batch, loss_mask=lossy & (at < density))
        loss, _ = graphed.train_step(one)
        loss, grads = float(loss), graphed.engine.flat_g.float().clone()
        with monkeypatch.context() as patched:
            patched.setattr(cls, "_takes_needed_rows", lambda *_: False)
            want, _ = eager.train_step(one)
            want, want_grads = float(want), eager.engine.flat_g.float().clone()
        assert len(graphed._graphed.cache) == 1
        assert abs(loss - want) <= 2e-4 * abs(want) + 1e-6, density
        # bf16 gradients, sums over rows and queries in another order
        assert torch.isfinite(grads).all() and float((grads - want_grads).norm()) <= 1e-2 * float(want_grads.norm()) + 1e-12, density
    ops.check_gemm_status()


@pytest.mark.gpu
@pytest.mark.parametrize("algorithm", ["eagle3", "mtp"])
def test_gpu_saved_tensor_hooks_get_tensors_of_the_batch(monkeypatch, algorithm):
    """A hook that packs what is saved by its largest value: no row may hold what nobody wrote."""
    if algorithm == "eagle3":
        model, batch = _model(1, 64, False, 688, True), _gpu_batch(2100, "spans")
        kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
    else:
        model = _mtp(0, 512, 64, 1000).cuda().bfloat16()
        batch = {"input_ids": torch.randint(0, 1000, (1, 1540)).cuda(), "hidden_states": torch.randn(1, 1540, 512).bfloat16().cuda(), "loss_mask": _mask("spans", 1540)[None].cuda()}
        kwargs = {"return_logits": False}
    largest = []

    def pack(t):
        if t.is_floating_point() and t.numel():
            largest.append(t.detach().abs().max())
        return t

    results = []
    for whole in (True, False):
        with monkeypatch.context() as patched:
            if whole:
                patched.setattr(type(model), "_takes_needed_rows", lambda *_: False)
            largest.clear()
            _poison()
            with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
                _, loss, _ = model(**batch, **kwargs)
            results.append(torch.stack([v.float() for v in largest]))
    assert torch.isfinite(results[0]).sum() == torch.isfinite(results[1]).sum() and results[0].shape == results[1].shape
    taken = []
    monkeypatch.setattr(ops, "step_rows", lambda *args, made=ops.step_rows, **kw: taken.append(1) or made(*args, **kw))
    model(**batch, **kwargs)
    assert taken


@pytest.mark.gpu
def test_gpu_forward_mode_is_refused_as_before(monkeypatch):
    from torch.autograd import forward_ad

    model, batch = _model(1, 64, False, 688, True), _gpu_batch(2100, "spans")
    kwargs, _ = Eagle3DraftModel.get_trainer_kwargs(loss_fn="kl_div", ttt_steps=3, ttt_step_loss_decay=0.8)
    states, losses = batch["verifier_last_hidden_states"], []
    for whole in (True, False):
        with monkeypatch.context() as patched, forward_ad.dual_level():
            if whole:
                patched.setattr(Eagle3DraftModel, "_takes_needed_rows", lambda *_: False)
            dual = forward_ad.make_dual(states, torch.ones_like(states))
            with pytest.raises(Exception, match="jvp"):
                model(**dict(batch, verifier_last_hidden_states=dual), **kwargs)
            with torch.no_grad():
                losses.append(float(model(**batch, **kwargs)[1]))  # without a tangent it runs
    assert abs(losses[0] - losses[1]) <= 2e-4 * abs(losses[0])
