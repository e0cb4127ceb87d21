"""Gradients of block-structured extra keys (one CTA per KV head and key tile, over the query heads of its group) against fp64."""

import pytest
import torch

from speculators_b200.ops import AttnSpec, masked_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("heads", "kv"), [(3, 3), (6, 2), (8, 2), (16, 2)])  # groups of 1, 3, 4, 8
@pytest.mark.parametrize(("blocks", "block"), [(1, 8), (16, 8), (17, 8), (9, 16)])  # one block, a whole tile, a block over, two tiles less 112 rows
@pytest.mark.parametrize("head_dim", [64, 128])
def test_gradients(heads, kv, blocks, block, head_dim):
    gen = torch.Generator().manual_seed(heads * 100 + blocks)
    n, context = (blocks + (64 if head_dim == 64 else 0)) * block, 150  # 64 wide: up to 512 rows run elsewhere
    draw = lambda *shape: torch.randn(*shape, generator=gen).to("cuda", torch.bfloat16)  # noqa: E731
    q, k, v, ke, ve, go = draw(n, heads, head_dim), draw(context, kv, head_dim), draw(context, kv, head_dim), draw(n, kv, head_dim), draw(n, kv, head_dim), draw(n, heads, head_dim)
    rows = torch.arange(n, device="cuda", dtype=torch.int32)
    hi = (rows // block * 9) % context
    spec = AttnSpec(lo=torch.zeros_like(hi), hi=hi, extra_idx=(rows[:, None] // block * block + torch.arange(block, device="cuda", dtype=torch.int32)).contiguous(),
                    extra_block=block)
    ke, ve = ke.requires_grad_(), ve.requires_grad_()
    masked_attention(q.requires_grad_(), k, v, spec, ke, ve).backward(go)
    again = torch.autograd.grad(masked_attention(q, k, v, spec, ke, ve), (ke, ve), go)
    assert torch.equal(again[0], ke.grad) and torch.equal(again[1], ve.grad)  # the heads of a group meet in a fixed order

    seen = torch.cat([torch.arange(context, device="cuda") < hi[:, None], rows[:, None] // block == rows // block], 1)
    group, scale = heads // kv, head_dim**-0.5
    for g in range(kv):
        want = {"k": 0.0, "v": 0.0}
        bound = {"k": 0.0, "v": 0.0}
        for h in range(g * group, (g + 1) * group):
            keys, values = torch.cat([k[:, g], ke[:, g]]).double(), torch.cat([v[:, g], ve[:, g]]).double()
            qh, d = q[:, h].double(), go[:, h].double()
            p = torch.softmax((qh @ keys.T * scale).masked_fill(~seen, float("-inf")), -1).detach()
            out = p @ values.detach()
            dp, delta = d @ values.detach().T, (d * out).sum(-1, keepdim=True)
            ds = p * (dp - delta)
            # rounded to bf16 (2^-8 relative): p and ds before their products, the output in delta, the gradient itself
            ds_off = 2.0**-8 * ds.abs() + p * 2.0**-8 * (d * out).abs().sum(-1, keepdim=True)
            want["v"] = want["v"] + (p.T @ d)[context:]
            want["k"] = want["k"] + scale * (ds.T @ qh.detach())[context:]
            bound["v"] = bound["v"] + 2.0**-8 * (p.T @ d.abs())[context:]
            bound["k"] = bound["k"] + scale * (ds_off.T @ qh.detach().abs())[context:]
        for name, grad in (("k", ke.grad), ("v", ve.grad)):
            worst = ((grad[:, g].double() - want[name]).abs() / (bound[name] + 2.0**-8 * want[name].abs() + 1e-4)).max().item()
            assert worst <= 1.0, (name, worst)
