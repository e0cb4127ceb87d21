"""Row bookkeeping kernels (document intervals, P-EAGLE sampling and mask, repeated rows, embedding gradients) against the
CPU formulations and fp32 autograd."""

import pytest
import torch

from speculators_b200 import ops
from speculators_b200.models.eagle3.attention import causal_document_interval
from speculators_b200.models.peagle.attention import peagle_attn_spec
from speculators_b200.models.peagle.data import generate_cod_sample_indices

pytestmark = pytest.mark.gpu


def _docs(T, n):
    cuts = torch.randint(0, T, (n,)).sort().values
    doc = torch.bucketize(torch.arange(T), cuts, right=True)
    doc[T - T // 9:] = -1
    return doc


# less than one vector, around the 8192 entries of a round, several rounds
@pytest.mark.parametrize("T,n", [(1, 1), (77, 3), (8192, 5), (8193, 40), (20001, 2)])
@pytest.mark.parametrize("window", [None, 50])
def test_document_interval(T, n, window):
    torch.manual_seed(T)
    doc = _docs(T, n)
    for a, b in zip(causal_document_interval(doc.cuda(), window), causal_document_interval(doc, window)):
        assert torch.equal(a.cpu(), b)


@pytest.mark.parametrize("T,share,max_anchors,filter_zero", [(1, 1.0, None, True), (300, 0.5, None, True), (300, 0.9, 40, False), (9000, 0.6, 4000, True), (64, 0.0, None, True)])
def test_sampler_and_mask(T, share, max_anchors, filter_zero, monkeypatch):
    torch.manual_seed(T)
    mask = (torch.rand(1, T) < share).float()
    doc = _docs(T, 4)

    def perm(n, device=None):
        g = torch.Generator().manual_seed(n)
        return torch.rand(n, generator=g).argsort().to(device)

    monkeypatch.setattr(torch, "randperm", perm)
    kw = dict(num_depths=6, max_anchors=max_anchors, filter_position_zero=filter_zero)
    a, d = generate_cod_sample_indices(T, mask.cuda(), **kw)
    ra, rd = generate_cod_sample_indices(T, mask, **kw)
    assert torch.equal(a.cpu(), ra) and torch.equal(d.cpu(), rd)
    for window, valid in ((None, None), (20, None), (None, torch.rand(len(ra)) < 0.8)):
        got = peagle_attn_spec(a, d, doc.cuda(), 6, window, None if valid is None else valid.cuda())
        want = peagle_attn_spec(ra, rd, doc, 6, window, valid)
        assert torch.equal(got.lo.cpu(), want.lo) and torch.equal(got.hi.cpu(), want.hi)
        assert (got.extra_idx is None) == (want.extra_idx is None)
        assert got.extra_idx is None or torch.equal(got.extra_idx.cpu(), want.extra_idx)


@pytest.mark.parametrize("T,n,hd,rot", [(1, 2, 64, 64), (130, 131, 128, 128), (300, 900, 128, 64), (40, 77, 256, 256)])
def test_repeated_rows(T, n, hd, rot):
    """Shared rows through heads and residual against the same rows laid out; the two gradient rows hold the sum to fp32's digits."""
    torch.manual_seed(n)
    heads = (4, 2, 2)
    src = torch.randn(T + 2, 8 * hd, device="cuda").bfloat16()
    src[T + 1] = src[T]
    pos = torch.randint(0, 500, (n,), device="cuda")
    angle = torch.rand(500, rot // 2, device="cuda")
    wa, wb = ((torch.rand(hd, device="cuda") + 0.5).bfloat16().requires_grad_() for _ in range(2))
    x = src.clone().requires_grad_()
    out = ops.norm_rope_heads(x, wa, wb, 1e-6, pos, angle.cos(), angle.sin(), heads, hd, rot, split=T, repeated=True)
    res = ops.repeat_rows(x, n)
    grads = [torch.randn(o.shape, device="cuda").bfloat16() for o in (*out, res)]
    torch.autograd.backward([*out, res], grads)

    xf = src.float().requires_grad_()
    wf = [w.detach().float().requires_grad_() for w in (wa, wb)]
    laid = torch.cat([xf[:T], xf[T:T + 1].expand(n - T, -1)])
    rotated, col = [], 0
    for h, w in zip(heads, (*wf, None)):
        b = laid[:, col: col + h * hd].reshape(n, h, hd)
        col += h * hd
        if w is not None:
            b = ops._rms_norm_ref(b, w, 1e-6)
            b = ops._rope_ref(b.reshape(n, -1), pos, angle.cos(), angle.sin(), h, hd, rot, 1.0).view(n, h, hd)
        rotated.append(b)
    want = (rotated[0], rotated[1][:T], rotated[1][T:], rotated[2][:T], rotated[2][T:], laid)
    torch.autograd.backward(want, [g.float() for g in grads])
    for a, b in zip((*out, res), want):
        assert a.shape == b.shape and (a.float() - b).abs().max() <= 0.02 * b.abs().max()
    scale = xf.grad.abs().max()
    assert (x.grad[:T].float() - xf.grad[:T]).abs().max() <= 0.02 * scale
    assert (x.grad[T].float() + x.grad[T + 1].float() - xf.grad[T]).abs().max() <= 0.02 * scale
    for a, b in zip((wa, wb), wf):
        assert (a.grad.float() - b.grad).abs().max() <= 0.02 * b.grad.abs().max() + 0.02


@pytest.mark.parametrize("n,H,vocab,padding", [(1, 8, 5, None), (700, 264, 50, 3), (64, 4096, 1000, None)])
@pytest.mark.parametrize("attached", [False, True])
def test_embedding_gradient(n, H, vocab, padding, attached):
    torch.manual_seed(n)
    w = torch.randn(vocab, H, device="cuda").bfloat16().requires_grad_()
    if attached:
        w._flat_grad, w._grad_fresh = torch.full_like(w, float("nan")), True
    ids = torch.randint(0, vocab, (n,), device="cuda")
    d = torch.randn(n, H, device="cuda").bfloat16()
    wf = w.detach().float().requires_grad_()
    for _ in range(2):
        ops.embedding(ids, w, padding).backward(d)
        torch.nn.functional.embedding(ids, wf, padding).backward(d.float())
    got = w._flat_grad if attached else w.grad
    assert (got.float() - wf.grad).abs().max() <= 0.01 * wf.grad.abs().max()


# an id that fills a slice of 32 positions, crosses one edge, two, 8 and 9 (the last that a warp sums alone), many (a padded tail), more
# than 256 slices; H in part of a 128-column block
@pytest.mark.parametrize("lengths,H", [([32, 32, 1], 8), ([31, 257, 256, 288, 289, 33], 264), ([33, 31, 1], 136), ([1, 31, 64, 3, 70], 2056), ([5, 2048, 7, 300], 256), ([8300], 24), ([17] * 40, 128), ([8] * 3 + [8192], 64)])
@pytest.mark.parametrize("padding", [None, 1])
@pytest.mark.parametrize("attached", [False, True])
def test_embedding_gradient_of_frequent_ids(lengths, H, padding, attached):
    torch.manual_seed(H)
    ids = torch.repeat_interleave(torch.arange(len(lengths)) * 3, torch.tensor(lengths))[torch.randperm(sum(lengths))].cuda()
    w = torch.zeros(3 * len(lengths) + 1, H, device="cuda").bfloat16().requires_grad_()
    if attached:
        w._flat_grad, w._grad_fresh = torch.full_like(w, float("nan")), True
    d = torch.randn(ids.numel(), H, device="cuda").bfloat16()
    for _ in range(2):
        ops.embedding(ids, w, padding).backward(d)
    got = (w._flat_grad if attached else w.grad).double()
    keep = (ids != padding) if padding is not None else torch.ones_like(ids, dtype=torch.bool)
    want, size = (torch.zeros(w.shape, dtype=torch.double, device="cuda").index_add_(0, ids[keep], 2 * x.double()[keep]) for x in (d, d.abs()))
    # fp32 sums of at most max(lengths) terms; the sum is rounded to bf16, and so is its double
    assert ((got - want).abs() <= 2.0**-8 * want.abs() + max(lengths) * 2.0**-24 * size).all()


# ---- anchored blocks --------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("T,slots,block", [(1, 4, 8), (8, 4, 8), (9, 4, 8), (100, 200, 8), (700, 64, 16), (8192, 512, 8), (8193, 512, 16), (20000, 3000, 4)])
@pytest.mark.parametrize("density", [0.0, 0.02, 0.6, 1.0])
@pytest.mark.parametrize("distinct", [True, False])
def test_anchors_are_the_smallest_keys_in_order(T, slots, block, density, distinct):
    g = torch.Generator(device="cuda").manual_seed(T + slots)
    mask = torch.rand(T, generator=g, device="cuda") < density
    keys = torch.rand(T, generator=g, device="cuda")
    if not distinct:  # few keys: many equal the last one taken
        keys = (keys * 3).floor() / 3
    anchors, picked = ops.native().select_anchors(mask, keys, slots, block)
    valid = [i for i in range(max(T - block, 0)) if mask[i]] if T < 1000 else torch.nonzero(mask[: T - block]).flatten().tolist()
    k = keys.tolist()
    want = sorted(sorted(valid, key=lambda i: (k[i], i))[: min(slots, T)])
    assert anchors.tolist() == want + [0] * (slots - len(want)) and picked.tolist() == [True] * len(want) + [False] * (slots - len(want))


@pytest.mark.parametrize("window,non_causal", [(None, False), (5, False), (5, True), (10**6, False)])
@pytest.mark.parametrize("block", [1, 3, 8])
def test_anchor_specs_and_slots_match_their_definition(window, non_causal, block):
    from speculators_b200.models.dflash.attention import anchor_block_attn_spec

    T, mask_token = 90, 77
    doc = torch.tensor([0] * 20 + [1] * 31 + [2] * 29 + [-1] * 10)
    anchors, picked = torch.tensor([0, 3, 19, 20, 50, 79, 81, 89, 0, 0]), torch.tensor([True] * 8 + [False] * 2)
    want = anchor_block_attn_spec(doc, anchors, block, window, non_causal)
    got = anchor_block_attn_spec(doc.cuda(), anchors.cuda(), block, window, non_causal)
    for a, b in ((got.lo, want.lo), (got.hi, want.hi), (got.extra_idx, want.extra_idx)):
        assert a.dtype == b.dtype and torch.equal(a.cpu(), b)
    assert (got.extra_block, got.extra_block_causal) == (want.extra_block, want.extra_block_causal)

    ids, positions, mask = torch.arange(T) * 3 + 1, torch.arange(T) % 31, torch.arange(T) % 4 != 1
    index = (anchors[:, None] + torch.arange(block)).reshape(-1)
    for from_anchor in (False, True):
        token = torch.full((len(index),), mask_token)
        token[::block] = ids[anchors]
        counts = mask[index % T] & picked.repeat_interleave(block) & (index < T)
        if not from_anchor:
            counts[::block] = False
        want = token, (positions[anchors][:, None] + torch.arange(block)).reshape(-1), index, (index if from_anchor else index - 1) % T, counts
        got = ops.native().anchor_slots(anchors.cuda(), picked.cuda(), ids.cuda(), positions.cuda(), mask.cuda(), block, mask_token, from_anchor)
        assert all(torch.equal(a.cpu(), b) for a, b in zip(got, want))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float64])
def test_anchors_are_chosen_under_another_default_type(dtype):
    from speculators_b200.models.dflash.utils import select_anchors

    mask = torch.zeros(1, 50, dtype=torch.bool, device="cuda")
    mask[0, [3, 7, 30, 45]] = True
    torch.set_default_dtype(dtype)
    try:
        anchors, picked = select_anchors(mask, 5, 8)
    finally:
        torch.set_default_dtype(torch.float32)
    assert anchors.tolist() == [3, 7, 30, 0, 0] and picked.tolist() == [True] * 3 + [False] * 2


@pytest.mark.parametrize("window", [0, 1, -1, -3, 2**40])
@pytest.mark.parametrize("non_causal", [False, True])
def test_anchor_specs_of_any_window(window, non_causal):
    from speculators_b200.models.dflash.attention import anchor_block_attn_spec

    doc, anchors = torch.tensor([0] * 20 + [1] * 31 + [-1] * 10), torch.tensor([0, 3, 19, 20, 50, 55])
    want = anchor_block_attn_spec(doc, anchors, 4, window, non_causal)
    got = anchor_block_attn_spec(doc.cuda(), anchors.cuda(), 4, window, non_causal)
    for a, b in ((got.lo, want.lo), (got.hi, want.hi), (got.extra_idx, want.extra_idx)):
        assert torch.equal(a.cpu(), b)


@pytest.mark.parametrize("T", [65536, 65537, 140000])
@pytest.mark.parametrize("density", [0.001, 0.6])
def test_anchors_of_long_rows(T, density, monkeypatch):
    from speculators_b200.models.dflash import utils

    mask = torch.rand(1, T, device="cuda") < density
    if T > 65536:  # one block is no match for a long row
        monkeypatch.setattr(utils.ops, "native", lambda: pytest.fail("a long row in one block"))
    torch.manual_seed(T)
    anchors, picked = utils.select_anchors(mask, 300, 8)
    torch.manual_seed(T)
    keys = torch.rand(T, device="cuda").where(mask[0] & (torch.arange(T, device="cuda") < T - 8), 2.0)
    want = torch.sort(torch.sort(keys, stable=True).indices[: min(300, int((keys < 2).sum()))]).values
    n = len(want)
    assert torch.equal(anchors[:n], want) and picked[:n].all() and not picked[n:].any() and not anchors[n:].any()
