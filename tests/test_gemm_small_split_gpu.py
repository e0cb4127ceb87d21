"""The GEMM's small-tile and split-contraction kernels (variants 10-13: 128x64 tiles on 1, 2, 4, 8 CTAs; 4, 5: pair tiles over
2, 4 pairs) at the edges of their tiles, against an fp32 matmul of the same operands."""

import pytest
import torch

from speculators_b200 import ops

pytestmark = pytest.mark.gpu

LAYOUTS = [(False, False), (False, True), (True, False), (True, True)]


@pytest.mark.parametrize("variant", [10, 11, 12, 13, 4, 5])
@pytest.mark.parametrize("a_mn,b_mn", LAYOUTS)
# one step, fewer steps than members (some have nothing to add), ragged edges of every kind, more steps than the ring holds
@pytest.mark.parametrize("M,N,K", [(128, 64, 128), (8, 8, 8), (136, 72, 200), (264, 328, 1160), (128, 256, 2048)])
def test_every_layout_and_epilogue(variant, a_mn, b_mn, M, N, K):
    torch.manual_seed(M + K)
    a = (torch.randn((K, M) if a_mn else (M, K), device="cuda") * 0.5).bfloat16()
    b = (torch.randn((K, N) if b_mn else (N, K), device="cuda") * 0.5).bfloat16()
    wide = torch.randn(M, N + 8, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = (a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t())
    for epilogue in (0, 1):
        buf = wide.clone()
        out = buf[:, :N]
        want = ref + (out.float() if epilogue else 0)
        ops.native().gemm_variant(a, b, out, epilogue, a_mn, b_mn, status, variant)
        first = buf.clone()
        if epilogue == 0:  # the order of the partial sums is fixed
            ops.native().gemm_variant(a, b, out, epilogue, a_mn, b_mn, status, variant)
            assert torch.equal(first, buf)
        assert int(status.item()) == 0
        assert (out.float() - want).abs().max() <= 0.01 * want.abs().max() + 0.02
        assert torch.equal(buf[:, N:], wide[:, N:])


@pytest.mark.parametrize("variant", [10, 12, 3, 4])
def test_unaligned_columns_and_residual(variant):
    M, N, K = 130, 77, 264
    torch.manual_seed(0)
    a, b = (torch.randn(M, K, device="cuda") * 0.5).bfloat16(), (torch.randn(N, K, device="cuda") * 0.5).bfloat16()
    res, out = torch.randn(M, N, device="cuda").bfloat16(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.native().gemm_tn_variant(a, b, out, res, 2, status, variant)
    want = a.float() @ b.float().t() + res.float()
    assert int(status.item()) == 0 and (out.float() - want).abs().max() <= 0.01 * want.abs().max() + 0.02
