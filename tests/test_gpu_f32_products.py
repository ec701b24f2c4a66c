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


def _within(hold, at, rows, cols):
    return hold[at:at + rows * cols].view(rows, cols)


@pytest.mark.parametrize("m", [1, 3, 5, 9, 16, 20])
@pytest.mark.parametrize("n,k", [(51, 260), (33, 259), (17, 1028), (9, 1031), (37, 2052), (7, 24600)])
@pytest.mark.parametrize("a_at,w_at", [(0, 0), (1, 0), (0, 3), (4, 8)])
def test_few_rows_between_values_that_are_no_numbers(m, n, k, a_at, w_at):
    """The kernel for few rows (inner sizes beyond 256): rows, columns, chunks and pieces that are filled up, with all of A resident
    and piece by piece (24,600 wide; 2,052 wide for nine rows and more), bases on and off a 16-byte boundary, rows whose pitch is
    no multiple of one.  NaN in front of and behind both operands and the result must stay where it is."""
    from dryft_b200.ops import kernels as K

    pad = 64 * k
    hold_a, hold_w = (torch.full((pad + at + rows * k + pad,), float("nan"), device="cuda") for rows, at in ((m, a_at), (n, w_at)))
    hold_o = torch.full((8 + m * n + 1024,), float("nan"), device="cuda")
    a, w, out = _within(hold_a, pad + a_at, m, k), _within(hold_w, pad + w_at, n, k), _within(hold_o, 8, m, n)
    a.copy_(torch.randint(-3, 4, (m, k), device="cuda"))
    w.copy_(torch.randint(-3, 4, (n, k), device="cuda"))
    K.gemm_nt_f32(a, w, out)
    assert torch.equal(out.double(), a.double() @ w.double().T)          # whole numbers below 2^24: exact in any order
    assert bool(hold_o[:8].isnan().all()) and bool(hold_o[8 + m * n:].isnan().all())


@pytest.mark.parametrize("m", [1, 4, 8, 16])
@pytest.mark.parametrize("k", [320, 1024, 2048, 2050])
def test_overlapped_products_wait_for_one_another(m, k):
    """A chain of products that read one another's results, each launched over the tail of the one before: the bits of the same
    chain without overlap, eager and captured."""
    from dryft_b200.ops import kernels as K

    ws = [torch.randn(k, k, device="cuda") * k ** -0.5 for _ in range(6)]
    x0, bufs = torch.randn(m, k, device="cuda"), [torch.empty(m, k, device="cuda") for _ in range(2)]

    def chain(pdl):
        x = x0
        for i in range(18):
            K.gemm_nt_f32(x, ws[i % 6], bufs[i % 2], pdl=pdl)
            x = bufs[i % 2]
        return x

    want = chain(False).clone()
    assert bool(torch.isfinite(want).all())
    for b in bufs:
        b.fill_(float("nan"))
    assert torch.equal(chain(True), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(True)
    for _ in range(3):
        for b in bufs:
            b.fill_(float("nan"))
        graph.replay()
        assert torch.equal(got, want)
