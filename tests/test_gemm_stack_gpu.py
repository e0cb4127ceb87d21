"""Stacks of products with scaled epilogues and symmetric results (what the Newton-Schulz iteration of Muon runs on), against
fp32 matmuls, and the stacked iteration against the single-matrix one."""

import pytest
import torch

from speculators_b200 import ops
from speculators_b200.parallel.engine import _newton_schulz, _newton_schulz_stack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
# one tile, ragged tiles (the next matrix of the stack must not leak in), several pair tiles, a long contraction (split kernels)
@pytest.mark.parametrize("B,M,N,K", [(1, 64, 64, 64), (3, 136, 72, 200), (2, 776, 1032, 520), (2, 264, 256, 6144)])
def test_scaled_products_of_a_stack(B, M, N, K, a_mn, b_mn):
    torch.manual_seed(B + M)
    a = (torch.randn((B, K, M) if a_mn else (B, M, K), device="cuda") * 0.3).bfloat16()
    b = (torch.randn((B, K, N) if b_mn else (B, N, K), device="cuda") * 0.3).bfloat16()
    add = torch.randn(B, M, N, device="cuda").bfloat16()
    out = torch.empty(B, M, N, device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = (a.float().transpose(1, 2) if a_mn else a.float()) @ (b.float() if b_mn else b.float().transpose(1, 2))
    ops.native().gemm_stack(a, b, out, add, a_mn, b_mn, 0.7, -1.3, False, status)
    want = 0.7 * ref - 1.3 * add.float()
    assert int(status.item()) == 0 and (out.float() - want).abs().max() <= 0.01 * want.abs().max()


@pytest.mark.parametrize("B,M,K", [(1, 256, 128), (3, 264, 512), (2, 1024, 640), (1, 4096, 256)])
def test_symmetric_products_mirror_their_tiles(B, M, K):
    torch.manual_seed(M)
    x = (torch.randn(B, K, M, device="cuda") * 0.3).bfloat16()
    out = torch.empty(B, M, M, device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.native().gemm_stack(x, x, out, None, True, True, 1.0, 0.0, True, status)
    want = x.float().transpose(1, 2) @ x.float()
    assert int(status.item()) == 0 and (out.float() - want).abs().max() <= 0.01 * want.abs().max()
    assert torch.equal(out, out.transpose(1, 2))


@pytest.mark.parametrize("rows,cols", [(512, 256), (264, 1032), (128, 128)])
@pytest.mark.parametrize("steps", [4, 5])
def test_stacked_iteration_matches_the_single_one(rows, cols, steps):
    torch.manual_seed(rows)
    x = torch.randn(3, rows, cols, device="cuda")
    x = (x / x.flatten(1).norm(dim=1).view(-1, 1, 1)).bfloat16()
    work, other = x.clone(), torch.empty_like(x)
    _newton_schulz_stack(work, other, steps)
    got = other if steps % 2 else work
    for z in range(3):
        single = _newton_schulz(x[z], steps, normalise=False)  # the same roundings; products may be split differently
        assert (got[z].float() - single.float()).norm() <= 0.02 * single.float().norm()
        want = _newton_schulz(x[z].float().cpu(), steps, normalise=False)
        assert (got[z].float().cpu() - want).norm() <= 0.03 * want.norm()
