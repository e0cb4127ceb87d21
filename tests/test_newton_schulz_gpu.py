"""Newton-Schulz stacks against the same polynomial iteration in fp64: one iteration at a time and two on one Gram matrix,
the polynomial rounded once."""

import pytest
import torch

from speculators_b200 import ops
from speculators_b200.parallel import engine

pytestmark = pytest.mark.gpu


def _exact(x, steps):
    x = x.double()
    tall = x.shape[-2] > x.shape[-1]
    eye = torch.eye(min(x.shape[-2:]), dtype=x.dtype, device=x.device)
    for _ in range(steps):
        g = x.mT @ x if tall else x @ x.mT
        p = 3.4445 * eye - 4.7750 * g + 2.0315 * g @ g
        x = x @ p if tall else p @ x
    return x


@pytest.mark.parametrize("rows,cols", [(256, 256), (264, 520), (136, 1032), (1032, 136), (2000, 64), (64, 20000)])
@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("decades", [0, 2])
def test_stack_against_fp64(rows, cols, steps, decades, monkeypatch):
    monkeypatch.setattr(engine, "_NS_ONCE_FROM", 1)
    g = torch.Generator(device="cuda").manual_seed(rows + steps)
    x = torch.randn(2, rows, cols, generator=g, device="cuda", dtype=torch.float64)
    if decades:  # singular values over two decades
        u, _, vt = torch.linalg.svd(x, full_matrices=False)
        x = u * torch.logspace(0, -decades, min(rows, cols), device="cuda", dtype=torch.float64) @ vt
    x = (x / x.flatten(1).norm(dim=1).view(-1, 1, 1)).bfloat16()
    want = _exact(x, steps)
    work, other = x.clone(), torch.empty_like(x)
    engine._newton_schulz_stack(work, other, steps)
    got = (other if steps % 2 else work).double()
    # A step multiplies small singular values, and with them what rounding to bf16 (2^-9) left, by up to 3.44; large ones come near
    # the polynomial's flat part.  With every sum rounded on its own the iteration is 0.02 to 0.045 off after five steps.
    assert float((got - want).norm() / want.norm()) <= (0.02 if not decades else 0.045)


def test_diagonal_is_added_before_the_one_rounding():
    x = (torch.randn(2, 264, 264, device="cuda") * 0.1).bfloat16()
    out, status = torch.empty_like(x), ops.gemm_status(x.device)
    ops.native().gemm_stack(x, x, out, x, False, False, 0.5, -1.5, False, status, 2.25)
    want = 0.5 * x.double() @ x.double().mT - 1.5 * x.double() + 2.25 * torch.eye(264, device="cuda", dtype=torch.float64)
    assert float(((out.double() - want).abs() / want.abs().clamp(min=1e-2)).max()) <= 2**-8 and int(status) == 0


@pytest.mark.parametrize("rows,cols", [(2048, 6144), (8192, 2048), (3072, 4096)])
@pytest.mark.parametrize("share,low", [(0.1, 0.1), (1 / 16, 0.2), (0.5, 0.5)])
def test_wide_stacks_are_no_further_off_than_with_sums_rounded_on_their_own(rows, cols, share, low, monkeypatch):
    """A share of the singular values at one, the others lower."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    short, long = min(rows, cols), max(rows, cols)
    u, v = (torch.linalg.qr(torch.randn(n, short, generator=g, device="cuda", dtype=torch.float64))[0] for n in (short, long))
    x = (u * torch.where(torch.arange(short, device="cuda") < share * short, 1.0, low)) @ v.mT
    x = ((x if rows < cols else x.mT) / x.norm()).bfloat16()[None].contiguous()
    want = _exact(x, 5)

    def off():
        work, other = x.clone(), torch.empty_like(x)
        engine._newton_schulz_stack(work, other, 5)
        return float((other.double() - want).norm() / want.norm())

    now = off()
    monkeypatch.setattr(engine, "_NS_ONCE_FROM", 1 << 30)
    assert now <= off()


@pytest.mark.parametrize("batch,n", [(1, 2048), (2, 2048), (1, 2056), (1, 3072)])
def test_symmetric_polynomial_on_pair_tiles(batch, n):
    """Sizes that take tiles of 256 x 256: addends a tile ahead, mirrored stores, a diagonal in both halves, at 3072 divided tiles."""
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    x = torch.randn(batch, n, n, generator=g, device="cuda") * 0.02
    x = (x + x.mT).bfloat16()
    out, status = torch.empty_like(x), ops.gemm_status(x.device)
    ops.native().gemm_stack(x, x, out, x, False, False, 2.0315, -4.7750, True, status, 3.4445)
    eye = 3.4445 * torch.eye(n, device="cuda", dtype=torch.float64)
    want = 2.0315 * x.double() @ x.double() - 4.7750 * x.double() + eye
    size = 2.0315 * x.double().abs() @ x.double().abs() + 4.7750 * x.double().abs() + eye
    # one rounding to bf16, and n terms added in fp32
    assert ((out.double() - want).abs() <= 2.0**-8 * want.abs() + n * 2.0**-24 * size).all() and int(status) == 0
