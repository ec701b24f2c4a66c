"""The 32-bit product at the edges of its kernels: row counts around those where another kernel or another number of rows a
block takes over, inner sizes around a chunk, a piece and a slice, rows that are not 16-byte aligned."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 16, 17, 33, 65, 200])
@pytest.mark.parametrize("n,k", [(1, 3), (63, 64), (65, 66), (1000, 516), (70, 1024), (130, 1092), (40, 2052), (24, 9728), (33, 4099)])
def test_every_kernel_against_64_bits_and_against_one_row_alone(m, n, k):
    from dryft_b200.ops import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(m * 1009 + n * 31 + k)
    a, w = (torch.randn(r, k, generator=gen, device="cuda") for r in (m, n))
    out = torch.full((m, n), float("nan"), device="cuda")
    K.gemm_nt_f32(a, w, out)
    exact = a.double() @ w.double().T
    # a chunk's 64 additions and products, then one addition a chunk, each off by half a unit of its result at most
    bound = (65 + (k + 63) // 64) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - exact).abs() <= bound).all())
    for row in {0, m // 2, m - 1}:
        one = torch.empty(1, n, device="cuda")
        K.gemm_nt_f32(a[row:row + 1].contiguous(), w, one)
        assert torch.equal(one[0], out[row])


def test_values_outside_the_operands_are_never_read():
    """Rows and columns around the operands hold NaN: padding of tiles, pieces and row groups has to be zeros instead."""
    from dryft_b200.ops import kernels as K

    for m, n, k in [(3, 50, 68), (20, 50, 68), (100, 130, 100)]:
        hold_a, hold_w = torch.full(((m + 64) * k,), float("nan"), device="cuda"), torch.full(((n + 64) * k,), float("nan"), device="cuda")
        a, w = hold_a[:m * k].view(m, k), hold_w[:n * k].view(n, k)
        a.fill_(1.0)
        w.fill_(2.0)
        out = torch.empty(m, n, device="cuda")
        K.gemm_nt_f32(a, w, out)
        assert torch.equal(out, torch.full_like(out, 2.0 * k))
