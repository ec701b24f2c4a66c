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
