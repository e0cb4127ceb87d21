"""RMSNorm variants against fp32: zero-centred weights, the residual gradient added in the backward kernel, rows up to 32768,
the weight gradient alone, and gradients that go into an attached flat buffer."""

import pytest
import torch

from speculators_b200 import ops

pytestmark = pytest.mark.gpu


def _reference(x, w, eps, centred):
    xf = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)
    return xf * (1 + w if centred else w)


# narrow rows, one block per row at every register budget, the widest rows; one row and more rows than blocks
@pytest.mark.parametrize("rows,H", [(1, 8), (700, 128), (300, 264), (33, 4104), (50, 9000), (40, 16392), (700, 24576), (3, 32768)])
@pytest.mark.parametrize("centred", [False, True])
@pytest.mark.parametrize("input_grad", [True, False])
def test_fork_backward(rows, H, centred, input_grad):
    torch.manual_seed(H)
    x = torch.randn(rows, H, device="cuda").bfloat16().requires_grad_(input_grad)
    w = (torch.rand(H, device="cuda") - (0.5 if centred else -0.5)).bfloat16().requires_grad_()
    dy, dres = torch.randn(rows, H, device="cuda").bfloat16(), torch.randn(rows, H, device="cuda").bfloat16()
    y, res = ops.rms_norm_fork(x, w, 1e-5, centred)
    torch.autograd.backward([y, res] if input_grad else [y], [dy, dres] if input_grad else [dy])
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yf = _reference(xf, wf, 1e-5, centred)
    yf.backward(dy.float())
    assert (y.float() - yf).abs().max() <= 0.02 * yf.abs().max()
    assert (w.grad.float() - wf.grad).abs().max() <= 0.01 * wf.grad.abs().max() + 0.02
    if input_grad:
        want = xf.grad + dres.float()
        assert (x.grad.float() - want).abs().max() <= 0.02 * want.abs().max()


def test_weight_gradient_goes_to_the_flat_buffer():
    torch.manual_seed(0)
    x = torch.randn(100, 512, device="cuda").bfloat16()
    w = torch.ones(512, device="cuda", dtype=torch.bfloat16).requires_grad_()
    w._flat_grad, w._grad_fresh = torch.full_like(w, float("nan")), True  # the first gradient is stored, the second added
    dy = torch.randn_like(x)
    for _ in range(2):
        ops.rms_norm(x, w, 1e-5).backward(dy)
    xf = x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-5)
    want = 2 * (dy.float() * xf).sum(0)
    assert w.grad is None and (w._flat_grad.float() - want).abs().max() <= 0.02 * want.abs().max()


def test_eagle3_input_adds_the_half_gradient():
    torch.manual_seed(0)
    T, H = 130, 256
    e, h = torch.randn(T, H, device="cuda").bfloat16(), torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    we, wh = (torch.rand(H, device="cuda").bfloat16().requires_grad_() for _ in range(2))
    out, half = ops.eagle3_input_concat(e, h, we, wh, 1e-5, return_hidden_half=True)
    d, dh = torch.randn_like(out), torch.randn(T, H, device="cuda").bfloat16()
    torch.autograd.backward([out, half], [d, dh])
    hf, wf = h.detach().float().requires_grad_(), wh.detach().float().requires_grad_()
    _reference(hf, wf, 1e-5, False).backward(d[:, H:].float() + dh.float())
    assert (h.grad.float() - hf.grad).abs().max() <= 0.02 * hf.grad.abs().max() + 0.02
    assert (wh.grad.float() - wf.grad).abs().max() <= 0.02 * wf.grad.abs().max() and torch.isfinite(we.grad).all()


@pytest.mark.parametrize("hd,rot,T", [(64, 64, 1), (128, 128, 700), (256, 64, 77)])
@pytest.mark.parametrize("heads,split", [((3, 0, 0), None), ((2, 0, 2), 5), ((4, 2, 2), None), ((6, 1, 1), 40)])
def test_norm_rope_heads_has_the_bits_of_the_separate_steps(hd, rot, T, heads, split):
    torch.manual_seed(hd)
    split = min(split, T) if split is not None else None
    src = torch.randn(T, sum(heads) * hd, device="cuda").bfloat16()
    angle = torch.rand(300, rot // 2, device="cuda")
    pos = torch.randint(0, 300, (T,), device="cuda")
    weights = [(torch.rand(hd, device="cuda") + 0.5).bfloat16() for _ in range(2)]

    def run(fused):
        x, wa, wb = (t.clone().requires_grad_() for t in (src, *weights))
        args = (wa, wb if heads[1] else None, 1e-6, pos, angle.cos(), angle.sin(), heads, hd, rot, split)
        if fused:
            out = ops.norm_rope_heads(x, *args)
        else:
            blocks, col = [], 0
            for n, w in zip(heads, (wa, wb, None)):
                b = x[:, col: col + n * hd].reshape(T, n, hd) if n else None
                col += n * hd
                if n and w is not None:
                    b = ops.rope_(ops.rms_norm(b, w, 1e-6).reshape(T, n * hd), pos, angle.cos(), angle.sin(), n, hd, rot).view(T, n, hd)
                blocks.append(b)
            out = ops._head_blocks(blocks, split)
        g = torch.Generator(device="cuda").manual_seed(1)
        torch.autograd.backward(out, [torch.randn(o.shape, device="cuda", generator=g).bfloat16() for o in out])
        return [*out, x.grad, wa.grad, *([wb.grad] if heads[1] else [])]

    for a, b in zip(run(True), run(False), strict=True):
        assert torch.equal(a, b)


def test_row_slices_of_a_flat_gradient_are_stored_then_added():
    torch.manual_seed(0)
    w = torch.randn(384, 256, device="cuda").bfloat16().requires_grad_()
    w._flat_grad, w._grad_fresh = torch.full_like(w, float("nan")), True
    x = torch.randn(200, 256, device="cuda").bfloat16()
    want = torch.zeros(384, 256, device="cuda")
    for r0, r1 in ((128, 256), (0, 128), (128, 256)):
        dy = torch.randn(200, r1 - r0, device="cuda").bfloat16()
        ops.linear(x, w, rows=(r0, r1)).backward(dy)
        want[r0:r1] += dy.float().t() @ x.float()
    assert torch.isnan(w._flat_grad[256:]).all()
    ops.clear_fresh_grad(w)
    assert (w._flat_grad[256:] == 0).all() and (w._flat_grad.float() - want).abs().max() <= 0.02 * want.abs().max()


@pytest.mark.parametrize("rows,K,N", [(64, 128, 128), (1001, 512, 768), (300, 1536, 2048)])
def test_weight_gradients_beside_the_backward_pass(rows, K, N):
    """Several uses of a weight, a gradient that reaches it another way, and a pass that ends in an exception."""
    torch.manual_seed(rows)
    w = torch.randn(N, K, device="cuda").bfloat16().requires_grad_()
    x = torch.randn(rows, K, device="cuda").bfloat16().requires_grad_()
    w._flat_grad, w._grad_fresh = torch.full_like(w, float("nan")), True
    w.grad = w._flat_grad

    def hook(g):
        ops.clear_fresh_grad(w)
        return g

    w.register_hook(hook)
    stop = ops.linear(x, w)
    stop.register_hook(lambda g: (_ for _ in ()).throw(RuntimeError("stop")))
    with pytest.raises(RuntimeError, match="stop"):
        (ops.linear(stop.new_ones(rows, K) * 0, w).sum() + stop.sum()).backward()
    w._grad_fresh = True
    y = ops.linear(x, w)
    z = ops.linear(y[:, :K].contiguous(), w) if N >= K else y
    (z.float().pow(2).mean() + (w.float() * 0.5).sum()).backward()
    got = w._flat_grad.float()
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yf = xf @ wf.t()
    zf = yf[:, :K].bfloat16().float().detach() + (yf[:, :K] - yf[:, :K].detach())
    zf = zf @ wf.t() if N >= K else yf
    (zf.pow(2).mean() + (wf * 0.5).sum()).backward()
    assert (got - wf.grad).abs().max() <= 0.02 * wf.grad.abs().max()


@pytest.mark.parametrize("rows,H", [(1, 264), (77, 1024), (2368, 4096), (2369, 4096), (3000, 4104), (900, 8192), (901, 12296), (700, 24576)])
def test_a_sum_and_its_norm_in_one_launch_give_the_same_bits(rows, H):
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, add, w = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((rows, H), (rows, H), (H,)))
    with torch.no_grad():
        total, normed = ops.add_rms_norm(x, add, w, 1e-6)
        assert torch.equal(total, x + add) and torch.equal(normed, ops.rms_norm(x + add, w, 1e-6))


@pytest.mark.parametrize("family,hd", [("llama", 64), ("llama", 128), ("qwen3", 128), ("qwen3", 256)])
@pytest.mark.parametrize("rows", [1, 100, 513, 2500])
def test_a_decoder_layer_in_one_call_gives_the_bits_of_its_modules(family, hd, rows, monkeypatch):
    from speculators_b200.verifier import tp

    cfg = {"architectures": ["LlamaForCausalLM"], "model_type": family, "hidden_size": 512, "num_hidden_layers": 3, "num_attention_heads": 4,
           "num_key_value_heads": 2, "head_dim": hd, "intermediate_size": 640, "vocab_size": 128, "rms_norm_eps": 1e-5, "rope_theta": 10000.0,
           "max_position_embeddings": 4096, "hidden_act": "silu"}
    verifier = tp.TensorParallelVerifier(cfg, seed=1, device="cuda", dtype=torch.bfloat16, resident=True)
    ids, doc = torch.randint(0, 128, (1, rows), device="cuda"), (torch.arange(rows, device="cuda") // 400).unsqueeze(0)
    taken = []
    fwd = tp.decoder_layer_fwd
    monkeypatch.setattr(tp, "decoder_layer_fwd", lambda *a: taken.append(fwd(*a)) or taken[-1])
    got = verifier.forward(ids, [0, 2], doc)
    assert len(taken) == 3 and all(t is not None for t in taken)
    monkeypatch.setattr(tp, "decoder_layer_fwd", lambda *a: None)
    want = verifier.forward(ids, [0, 2], doc)
    assert all(torch.equal(got[k], want[k]) for k in want)
    seen = []
    verifier._layers[1].mlp.down_proj.register_forward_hook(lambda m, i, o: seen.append(o.shape))  # its layer's modules are called
    monkeypatch.setattr(tp, "decoder_layer_fwd", fwd)
    again = verifier.forward(ids, [0, 2], doc)
    assert len(seen) == 1 and all(torch.equal(again[k], want[k]) for k in want)


@pytest.mark.parametrize("which", ["input_layernorm", "post_attention_layernorm"])
def test_a_layer_with_a_centred_norm_is_not_one_call_of_the_plain_one(which, monkeypatch):
    from speculators_b200.models.moe import ZeroCenteredRMSNorm
    from speculators_b200.verifier import tp

    cfg = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_size": 512, "num_hidden_layers": 3, "num_attention_heads": 4,
           "num_key_value_heads": 2, "head_dim": 128, "intermediate_size": 640, "vocab_size": 128, "rms_norm_eps": 1e-5, "rope_theta": 10000.0,
           "max_position_embeddings": 4096, "hidden_act": "silu"}
    verifier = tp.TensorParallelVerifier(cfg, seed=1, device="cuda", dtype=torch.bfloat16, resident=True)
    ids = torch.randint(0, 128, (1, 100), device="cuda")
    verifier.forward(ids, [0])
    setattr(verifier._layers[1], which, ZeroCenteredRMSNorm(512).to("cuda", torch.bfloat16))
    got = verifier.forward(ids, [0, 1, 2])
    monkeypatch.setattr(tp, "decoder_layer_fwd", lambda *a: None)
    want = verifier.forward(ids, [0, 1, 2])
    assert all(torch.equal(got[k], want[k]) for k in want)
