"""Row losses at the edges of their kernel: widths around the vectors and the block's stride, masked logits (the type's lowest
value, some -inf), equal maxima - against fp64."""

import pytest
import torch

from speculators_b200 import ops

pytestmark = pytest.mark.gpu

LOWEST = torch.finfo(torch.bfloat16).min


def _reference(op, x, t):
    lq, lp = torch.log_softmax(x.double(), -1), torch.log_softmax(t.double(), -1)
    p, q = lp.exp(), lq.exp()
    if op == "kl_div":
        return torch.where(p > 0, p * (lp - lq), 0.0).sum(-1)
    if op == "ce":
        return -lq.gather(-1, t.double().argmax(-1, keepdim=True)).squeeze(-1)
    return 1.0 - torch.minimum(p, q).sum(-1)


def _check(op, x, t):
    loss, am_d, am_t = ops.fused_row_loss(op, x, t)
    want = _reference(op, x, t)
    # sums of up to 5000 fp32 terms of magnitude up to the loss and the logits' spread (2^-24 each, and approximate exponentials)
    assert torch.allclose(loss.double(), want, rtol=2e-5, atol=2e-5), (loss.double() - want).abs().max()
    assert torch.equal(am_d, x.double().argmax(-1)) and torch.equal(am_t, t.double().argmax(-1))


@pytest.mark.parametrize("op", ["kl_div", "ce", "tv"])
@pytest.mark.parametrize("V", [1, 3, 8, 9, 2040, 2048, 2056, 4096, 4104, 4999, 5000])
def test_widths(op, V):
    g = torch.Generator(device="cuda").manual_seed(V)
    # distinct values in every row: a row has one maximum (bf16 holds 8 bits, so a permutation of few values would repeat)
    x, t = ((torch.randn(7, V, generator=g, device="cuda") * 3).bfloat16() for _ in range(2))
    rows = torch.arange(7, device="cuda")
    for m in (x, t):
        m[rows, torch.randint(0, V, (7,), generator=g, device="cuda")] = 20.0
    _check(op, x, t)


@pytest.mark.parametrize("op", ["kl_div", "ce", "tv"])
def test_masked_columns(op):
    V = 4104
    g = torch.Generator(device="cuda").manual_seed(1)
    x, t = (torch.randn(6, V, generator=g, device="cuda").bfloat16() for _ in range(2))
    keep = torch.rand(6, V, generator=g, device="cuda") < 0.3
    keep[1] = False  # one column left, behind the first vectors of all threads
    keep[1, 4101] = True
    keep[2, :2048] = False  # nothing in the first round of loads
    x[~keep], t[~keep] = LOWEST, LOWEST
    for m in (x, t):
        m[torch.arange(6), keep.int().argmax(-1)] = 9.0
    _check(op, x, t)


@pytest.mark.parametrize("op", ["kl_div", "ce", "tv"])
def test_infinite_logits_of_improbable_tokens(op):
    g = torch.Generator(device="cuda").manual_seed(4)
    x, t = ((torch.randn(5, 4104, generator=g, device="cuda") * 3).bfloat16() for _ in range(2))
    for m in (x, t):
        m[torch.arange(5), torch.tensor([3, 2050, 4103, 0, 4096])] = 20.0
    t[:, 1::3] = float("-inf")
    x[0, 1::3] = float("-inf")  # where the target's probability is zero too: nothing is lost there
    _check(op, x, t)


@pytest.mark.parametrize("V", [7, 512, 4104, 32000])
def test_divergence_and_variation_of_listed_target_rows_in_one_pass(V):
    g = torch.Generator(device="cuda").manual_seed(V)
    x, t = (torch.randn(n, V, generator=g, device="cuda").bfloat16().mul_(3) for n in (33, 9))
    to = torch.randint(0, 9, (33,), generator=g, device="cuda", dtype=torch.int32)
    active = torch.rand(33, generator=g, device="cuda") < 0.7
    x.requires_grad_(True)
    loss, am_d, am_t, tv = ops.fused_row_loss("kl_div", x, t, active=active, target_row=to, with_tv=True)
    loss.sum().backward()
    got, x.grad = x.grad, None
    rows = t[to.long()]
    want, want_d, want_t = ops.fused_row_loss("kl_div", x, rows, active=active)  # the same sums in the same order
    want.sum().backward()
    assert torch.equal(loss, want) and torch.equal(am_d, want_d) and torch.equal(am_t, want_t) and torch.equal(got, x.grad)
    assert torch.equal(tv, ops.fused_row_loss("tv", x.detach(), rows, active=active)[0]) and not tv.requires_grad


def test_the_first_of_equal_maxima():
    x = torch.zeros(4, 4100, device="cuda", dtype=torch.bfloat16)
    t = x.clone()
    for r, at in enumerate(([5, 6, 2050], [4099, 4098], [2055, 2049], [0, 4099])):
        x[r, at] = 7.0
        t[r, [a // 2 for a in at]] = 7.0
    _, am_d, am_t = ops.fused_row_loss("kl_div", x, t)
    assert am_d.tolist() == [5, 4098, 2049, 0] and am_t.tolist() == [2, 2049, 1024, 0]
