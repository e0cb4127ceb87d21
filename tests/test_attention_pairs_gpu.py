"""Attention forward, two query heads of a KV head per block: against the same heads run one per block (a shorter grid takes that
kernel), bit for bit, and against dense fp32 attention."""

import pytest
import torch

from speculators_b200 import ops
from speculators_b200.ops import AttnSpec

pytestmark = pytest.mark.gpu

HEADS, KV = 64, 8  # 64 heads x 7 query tiles and more: pairs; the 8 heads of one group: one head per block


def _intervals(T, documents, gen):
    lo = torch.zeros(T, dtype=torch.int32)
    hi = torch.arange(1, T + 1, dtype=torch.int32)
    for cut in sorted(torch.randperm(T - 1, generator=gen)[: documents - 1].add(1).tolist()):
        lo[cut:] = cut
    hi[T - 40 :] = lo[T - 40 :] = 0  # rows without a key
    return lo.cuda(), hi.cuda()


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("tokens", [769, 896, 1100])  # seven tiles, the last with one row; seven whole ones; nine
@pytest.mark.parametrize("extras", ["none", "rows", "block8", "block16_causal"])
def test_pairs_match_one_head_per_block(head_dim, tokens, extras):
    gen = torch.Generator().manual_seed(tokens + head_dim)
    draw = lambda *shape: torch.randn(*shape, generator=gen).to("cuda", torch.bfloat16)  # noqa: E731
    lo, hi = _intervals(tokens, 3, gen)
    block = {"block8": 8, "block16_causal": 16}.get(extras, 0)
    n = tokens - tokens % block if block else tokens
    q, k, v = draw(n, HEADS, head_dim), draw(tokens, KV, head_dim), draw(tokens, KV, head_dim)
    ke = ve = None
    spec = AttnSpec(lo=lo[:n].contiguous(), hi=hi[:n].contiguous())
    rows = torch.arange(n, device="cuda", dtype=torch.int32)
    if extras == "rows":
        ke, ve = draw(2 * n, KV, head_dim), draw(2 * n, KV, head_dim)
        idx = torch.stack([rows, rows + n], 1)
        idx[n // 2 :: 3, 1] = -1
        spec = AttnSpec(lo=spec.lo, hi=spec.hi, extra_idx=idx)
    elif block:
        ke, ve = draw(n, KV, head_dim), draw(n, KV, head_dim)
        idx = rows[:, None] // block * block + torch.arange(block, device="cuda", dtype=torch.int32)
        causal = extras.endswith("causal")
        if causal:
            idx = torch.where(idx <= rows[:, None], idx, -1)
        spec = AttnSpec(lo=spec.lo, hi=spec.hi, extra_idx=idx.contiguous(), extra_block=block, extra_block_causal=causal)
    with torch.no_grad():
        out = ops.masked_attention(q, k, v, spec, ke, ve)
        group = HEADS // KV
        for g in (0, KV - 1):
            take = lambda x: None if x is None else x[:, g : g + 1].contiguous()  # noqa: B023, E731
            alone = ops.masked_attention(q[:, g * group : (g + 1) * group].contiguous(), take(k), take(v), spec, take(ke), take(ve))
            assert torch.equal(out[:, g * group : (g + 1) * group], alone)
        # dense fp32: the probabilities that the kernel multiplies are bf16 and so is the output, up to 2^-8 relative each
        g, h = 3, 3 * group + 5
        keys, values = k[:, g].float(), v[:, g].float()
        at = torch.arange(tokens, device="cuda")
        seen = (at >= spec.lo[:, None]) & (at < spec.hi[:, None])
        if ke is not None:
            keys, values = torch.cat([keys, ke[:, g].float()]), torch.cat([values, ve[:, g].float()])
            more = torch.zeros(n, ke.shape[0] + 1, dtype=torch.bool, device="cuda")
            more.scatter_(1, torch.where(spec.extra_idx >= 0, spec.extra_idx, ke.shape[0]).long(), True)
            seen = torch.cat([seen, more[:, :-1]], 1)
        scores = (q[:, h].float() @ keys.T * head_dim**-0.5).masked_fill(~seen, float("-inf"))
        probs = torch.softmax(scores, -1).nan_to_num(0.0)
        want, bound = probs @ values, 2.0**-7 * (probs @ values.abs()) + 1e-6
        worst = ((out[:, h].float() - want).abs() / bound).max().item()
        assert worst <= 1.0, worst
