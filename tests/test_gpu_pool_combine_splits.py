"""Row-wise attention over pages in splits around those that the combining launch requests together (16) and weighs together (128): against
the plain softmax in 64-bit, with splits that have no keys and with a sink."""

import pytest
import torch

from test_gpu_kernels import DEV
from test_gpu_vobusun_parts import i32
from dryft_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d, dv, group", [(16, 16, 2), (24, 24, 1), (128, 128, 4), (192, 192, 1)])
@pytest.mark.parametrize("n_splits", [2, 15, 16, 17, 33, 128, 130])
def test_splits_joined(d, dv, group, n_splits):
    torch.manual_seed(n_splits)
    H, G, page, n = 4, 4 // group, 64, 3
    k, v = torch.randn(3, G, page, d, device=DEV), torch.randn(3, G, page, dv, device=DEV)
    table, pos = i32([[2, 0, 1]]), [0, 40, 190]
    q, sink = torch.randn(n, H, d, device=DEV), torch.tensor([0.5, -1.0, 3.0, 0.0], device=DEV)
    flat = lambda x: x[table[0].long()].permute(1, 0, 2, 3).reshape(G, 3 * page, -1).double().cpu()
    for s in (None, sink):
        out = torch.full((n, H, dv), float("nan"), device=DEV)
        po, pm = torch.full((n, H, n_splits, dv), float("nan"), device=DEV), torch.full((n, H, n_splits, 2), float("nan"), device=DEV)
        K.pool_attn_rows(q, k, v, table, None, s, i32([0] * n), i32(pos), out, 0.5, 1 << 30, 0, n_splits, po, pm)
        for t, p in enumerate(pos):
            for h in range(H):
                z = flat(k)[h // group, :p + 1] @ q[t, h].double().cpu() * 0.5
                if s is not None:
                    z = torch.cat([z, s[h:h + 1].double().cpu()])
                want = torch.softmax(z, 0)[:p + 1] @ flat(v)[h // group, :p + 1]
                # 32-bit scores of up to 192 terms (below 40) (their error goes into the exponents) and sums of 191 keys: 2e-5 of the values
                assert float((out[t, h].double().cpu() - want).abs().max()) <= 2e-5 * 4.0, (t, h)


@pytest.mark.parametrize("sink", [False, True])
def test_a_split_whose_scores_overflow_leaves_the_others_alone(sink):
    """The first 32 keys' scores are -inf in 32-bit; they are the whole of the first split, whose own sums are then no numbers."""
    d, H, page, n_splits = 16, 2, 64, 3
    torch.manual_seed(5)
    k, v = torch.randn(2, 1, page, d, device=DEV), torch.randn(2, 1, page, d, device=DEV)
    k[1, 0, :32] = -3e38
    q, s = torch.rand(1, H, d, device=DEV) + 0.5, torch.tensor([0.3, -0.7], device=DEV) if sink else None
    out = torch.full((1, H, d), float("nan"), device=DEV)
    po, pm = torch.full((1, H, n_splits, d), float("nan"), device=DEV), torch.full((1, H, n_splits, 2), float("nan"), device=DEV)
    K.pool_attn_rows(q, k, v, i32([[1, 0]]), None, s, i32([0]), i32([95]), out, 0.5, 1 << 30, 0, n_splits, po, pm)
    flat = lambda x: torch.cat([x[1, 0], x[0, 0]])[32:96].double().cpu()
    for h in range(H):
        z = flat(k) @ q[0, h].double().cpu() * 0.5
        if sink:
            z = torch.cat([z, s[h:h + 1].double().cpu()])
        want = torch.softmax(z, 0)[:64] @ flat(v)
        # 32-bit scores of 16 terms (below 20: their error goes into the exponents) and sums of 64 keys
        assert float((out[0, h].double().cpu() - want).abs().max()) <= 1e-5 * 4.0
