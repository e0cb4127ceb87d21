"""GEMMs that divide the tiles of a part-filled last wave between CTA pairs: every layout and epilogue at shapes that divide, against fp32
products of the same bf16 operands; repeats, streams and graph replays give the same bits."""

import pytest
import torch

from speculators_b200 import ops

pytestmark = pytest.mark.gpu

# 74 pairs, tiles of 256 x 256: (M, N, K) with the tile counts
SHAPES = [
    (1280, 4096, 4096),  # 80: one full wave and six tiles, four parts each
    (1203, 4104, 4096),  # 85, ragged on both edges
    (2304, 2304, 5000),  # 81, ragged contraction
    (512, 2048, 8192),  # 16: fewer tiles than pairs
    (1024, 4096, 14336),  # 64: two rounds, 37 tiles in two parts and 27 in two
    (2048, 4096, 14336),  # 128: a wave, 37 tiles in two parts and 17 in four
    (300, 256, 30000),  # 2, eight parts
    (4864, 4096, 4096),  # 304: four full waves and eight tiles
]


def _rand(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").bfloat16()


def _check(got, want):
    # fp32 accumulation, one rounding to bf16 (relative 2^-9 at most)
    assert float((got.float() - want).norm() / want.norm()) < 4e-3


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_layouts_and_epilogues(M, N, K):
    nat, status = ops.native(), ops.gemm_status(torch.device("cuda", 0))
    a, b, r = _rand(M, K, seed=1), _rand(N, K, seed=2), _rand(M, N, seed=3)
    want = a.float() @ b.float().T
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    nat.gemm_tn_variant(a, b, out, None, 0, status, 6)
    _check(out, want)
    nat.gemm_tn_variant(a, b, out, r, 2, status, 6)
    _check(out, want + r.float())
    out.copy_(r)
    nat.gemm_tn_variant(a, b, out, None, 1, status, 6)
    _check(out, want + r.float())
    if N % 8 == 0:
        nat.gemm_variant(a, b.T.contiguous(), out, 0, False, True, status, 6)
        _check(out, want)
    if M % 8 == 0:
        nat.gemm_variant(a.T.contiguous(), b.T.contiguous(), out, 0, True, True, status, 6)
        _check(out, want)
    assert int(status) == 0


@pytest.mark.parametrize("live", [256, 768, 1280])
def test_row_count_decides_on_the_device(live):
    a, b = _rand(1536, 4096, seed=1), _rand(4096, 4096, seed=2)
    a[live:] = float("nan")
    status, out = ops.gemm_status(a.device), torch.full((1536, 4096), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.native().gemm_tn_variant(a, b, out, None, 0, status, 6, torch.tensor([live], dtype=torch.int32, device="cuda"))
    _check(out[:live], a[:live].float() @ b.float().T)
    assert (out[live:] == 7.0).all() and int(status) == 0


def test_symmetric_stack():
    x = _rand(3, 2560, 2048, seed=1)  # 55 tiles on and above the diagonal, times three
    out, status = torch.empty(3, 2560, 2560, device="cuda", dtype=torch.bfloat16), ops.gemm_status(x.device)
    ops.native().gemm_stack(x, x, out, None, False, False, 1.0, 1.0, True, status)
    _check(out, x.float() @ x.float().transpose(1, 2))
    assert torch.equal(out, out.transpose(1, 2)) and int(status) == 0


def test_the_same_bits_from_every_launch_stream_and_replay():
    a, b = _rand(1280, 4096, seed=1), _rand(4096, 4096, seed=2)
    status = ops.gemm_status(a.device)

    def product():
        out = torch.empty(1280, 4096, device="cuda", dtype=torch.bfloat16)
        ops.native().gemm_tn_variant(a, b, out, None, 0, status, 6)
        return out

    want = product()
    assert all(torch.equal(product(), want) for _ in range(200))  # more launches than one slab of flags serves
    streams = [torch.cuda.Stream() for _ in range(2)]
    results = []
    torch.cuda.synchronize()
    for _ in range(40):  # at the same time on two streams
        for s in streams:
            with torch.cuda.stream(s):
                results.append(product())
    torch.cuda.synchronize()
    assert all(torch.equal(r, want) for r in results)
    graphs = []
    for _ in range(2):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [product() for _ in range(70)]
        graphs.append((graph, outs))
    for _ in range(3):
        for graph, outs in graphs:
            for o in outs:
                o.zero_()
            graph.replay()
            assert all(torch.equal(o, want) for o in outs)
            assert torch.equal(product(), want)
    assert int(status) == 0
