"""Fused mixture-of-experts call, gated attention kernels and the merged rotation gradient against fp32 / step-by-step forms."""

import pytest
import torch

from speculators_b200 import ops
from speculators_b200.models.moe import expert_forward
from speculators_b200.ops.moe import moe_experts, moe_experts_ok

pytestmark = pytest.mark.gpu


def _close(a, b, rel):
    assert (a.float() - b).abs().max() <= rel * b.abs().max() + 1e-3


# one slot; one expert takes everything; empty experts; segments that end on and beside a tile; the most experts
@pytest.mark.parametrize("T,E,k,spread", [(1, 4, 1, 4), (640, 3, 1, 1), (300, 64, 8, 40), (1025, 16, 2, 16), (257, 1024, 10, 1024)])
@pytest.mark.parametrize("shared", [False, True])
def test_experts(T, E, k, spread, shared):
    torch.manual_seed(T)
    H, I = 256, 256

    def leaf(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda") * scale).bfloat16().requires_grad_()

    x, gu, dn = leaf(T, H), leaf(E, 2 * I, H, scale=0.06), leaf(E, H, I, scale=0.06)
    top_e = torch.stack([torch.randperm(spread, device="cuda")[:k] for _ in range(T)]) if spread >= k else torch.zeros(T, k, device="cuda", dtype=torch.long)
    p = torch.rand(T, k, device="cuda").bfloat16().requires_grad_()
    extra = [leaf(T, H), leaf(T, 1), leaf(T, H)] if shared else [None, None, None]
    dn._flat_grad, dn._grad_fresh = torch.full_like(dn, float("nan")), True
    assert moe_experts_ok(x, gu, dn)
    out = moe_experts(x, p, top_e, gu, dn, *extra)
    dout = torch.randn(T, H, device="cuda").bfloat16()
    out.backward(dout)
    ops.check_gemm_status()

    inputs = [t for t in (x, p, gu, dn, *extra) if t is not None]
    ref = {id(t): t.detach().float().requires_grad_() for t in inputs}
    rows = ref[id(x)].repeat_interleave(k, 0)
    y = torch.zeros(T * k, H, device="cuda")
    for e in torch.unique(top_e).tolist():
        at = (top_e.reshape(-1) == e).nonzero().squeeze(1)
        y = y.index_put((at,), expert_forward(rows[at], torch.zeros(len(at), device="cuda", dtype=torch.long), ref[id(gu)][e:e + 1], ref[id(dn)][e:e + 1]))
    want = (y.view(T, k, H) * ref[id(p)].unsqueeze(-1)).sum(1)
    if shared:
        want = want + torch.sigmoid(ref[id(extra[1])]) * ref[id(extra[0])] + ref[id(extra[2])]
    want.backward(dout.float())
    _close(out, want, 0.02)
    for t in inputs:
        _close(dn._flat_grad if t is dn else t.grad, ref[id(t)].grad, 0.03)


@pytest.mark.parametrize("T,heads,hd", [(1, 1, 16), (77, 3, 128), (300, 16, 256)])
@pytest.mark.parametrize("merged", [True, False])  # the gate's gradient arrives inside the shared buffer, or on its own
def test_gated_query(T, heads, hd, merged):
    torch.manual_seed(hd)
    qg = torch.randn(T, heads, 2 * hd, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(hd, device="cuda") * 0.3).bfloat16().requires_grad_()
    att, dy, dq = (torch.randn(T, heads, hd, device="cuda").bfloat16().requires_grad_() for _ in range(3))
    q, gate = ops.split_gated_query(qg, w, 1e-6)
    y = ops.gated(att, gate if merged else gate * 1)
    torch.autograd.backward([q, y], [dq.detach(), dy.detach()])
    qf, wf, af = (t.detach().float().requires_grad_() for t in (qg, w, att))
    yf = af * torch.sigmoid(qf[..., hd:])
    nf = ops._rms_norm_ref(qf[..., :hd], wf, 1e-6, True)
    torch.autograd.backward([nf, yf], [dq.detach().float(), dy.detach().float()])
    for a, b in ((q, nf), (y, yf), (qg.grad, qf.grad), (w.grad, wf.grad), (att.grad, af.grad)):
        _close(a, b, 0.02)


@pytest.mark.parametrize("hd,rot", [(64, 64), (128, 128), (256, 64)])
@pytest.mark.parametrize("strided", [False, True])
def test_merged_rotation_gradient_has_the_bits_of_the_separate_steps(hd, rot, strided):
    torch.manual_seed(hd)
    T, nq, nk = 301, 4, 2
    make = (lambda n: torch.randn(T, n * hd + 8, device="cuda").bfloat16()[:, : n * hd]) if strided else (lambda n: torch.randn(T, n * hd, device="cuda").bfloat16())
    dq, dk, dv = make(nq), make(nk), make(nk)
    angle = torch.rand(400, rot // 2, device="cuda")
    pos = torch.randint(0, 400, (T,), device="cuda")
    args = (pos, angle.cos(), angle.sin())
    nat = ops.native()
    want = torch.cat([dq, dk, dv], -1)
    nat.rope_(want, *args, nq + nk, hd, rot, -1.0)
    assert torch.equal(nat.rope_merge(dq, dk, dv, True, *args, hd, rot, -1.0), want)
    want = dq.contiguous().clone()
    nat.rope_(want, *args, nq, hd, rot, -1.0)
    assert torch.equal(nat.rope_merge(dq, None, None, False, *args, hd, rot, -1.0), want)


@pytest.mark.parametrize("E", [1, 31, 64, 65, 256, 512, 1000])
@pytest.mark.parametrize("ties", [False, True])
def test_topk_rows(E, ties):
    g = torch.Generator(device="cuda").manual_seed(E)
    p = torch.randn(37, E, generator=g, device="cuda")
    if ties:
        p = (p * 2).round()
        p[0], p[1, E // 2], p[2, 0] = 0.0, float("nan"), float("-inf")
    for k in {1, min(E, 10), min(E, 32)}:
        got = ops.native().topk_rows(p, k)
        keyed = torch.where(p.isnan(), torch.full_like(p, float("inf")), p)
        assert torch.equal(got, torch.sort(keyed, dim=-1, descending=True, stable=True).indices[:, :k])


@pytest.mark.parametrize("E,k", [(16, 4), (256, 10)])
def test_equal_experts_are_chosen_in_the_order_of_topk(E, k):
    from speculators_b200.layer_config import TransformerLayerConfig
    from speculators_b200.models.moe import SparseMoeBlock

    cfg = TransformerLayerConfig(hidden_size=256, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2, head_dim=64, intermediate_size=256,
                                 vocab_size=512, model_type="qwen3_next", num_experts=E, num_experts_per_tok=k, moe_intermediate_size=128)
    torch.manual_seed(E)
    block = SparseMoeBlock(cfg).cuda().bfloat16()
    with torch.no_grad():
        block.gate.weight[1::2] = block.gate.weight[::2]  # each probability twice
        x = torch.randn(300, 256, device="cuda").bfloat16()
        want = torch.topk(torch.softmax(block.gate(x).float(), -1), k, dim=-1).indices
        assert torch.equal(block.route(x)[1], want)
