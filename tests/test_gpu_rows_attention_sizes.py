"""Row-wise attention at head sizes around those at which a thread of the combining launch takes one dim more, with one block a row, few
splits and more splits than keys, over pages of 64 and of 32, against 32-bit attention over the same keys."""

import math

import pytest
import torch

from test_gpu_kernels import DEV, K, _attn_ref, _fill_cache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n_heads,n_kv,d,page", [(torch.float32, 2, 2, 112, 64), (torch.bfloat16, 4, 1, 128, 32), (torch.float32, 4, 2, 144, 64),
                                                       (torch.bfloat16, 2, 2, 240, 64), (torch.float32, 2, 1, 256, 32)])
def test_head_sizes_of_the_combining_launch(dtype, n_heads, n_kv, d, page):
    k, scale, g = K(), 1.0 / math.sqrt(d), torch.Generator().manual_seed(d)
    positions = [0, 15, 33, 150, 299]
    n = len(positions)
    seqs = {i: (torch.randn(p + 1, n_kv, d, generator=g).to(dtype), torch.randn(p + 1, n_kv, d, generator=g).to(dtype)) for i, p in enumerate(positions)}
    q = torch.randn(n + 1, n_heads, d, generator=g).to(dtype)
    kc, vc, pt = _fill_cache(seqs, n_kv, d, page, dtype, n_pages=40, max_pages=10, slots=n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    for splits in (1, 3, 17, 131):
        out = torch.full((n + 1, n_heads * d), 9.0, device=DEV, dtype=dtype)
        po = torch.full((n + 1, n_heads, splits, d), float("nan"), device=DEV)
        pm = torch.full((n + 1, n_heads, splits, 2), float("nan"), device=DEV)
        k.attn_rows(q.to(DEV), kc, vc, pt, i32([*range(n), -1]), i32([*positions, 0]), out, scale, None, splits, po, pm)
        got = out.cpu().float()
        assert torch.count_nonzero(got[n]) == 0
        for i, p in enumerate(positions):
            want = _attn_ref(q[i], *seqs[i], p, scale, None)
            # 32-bit sums of up to 256 and 300 terms in other orders, then one rounding to the type of the result
            most = float(seqs[i][1].float().abs().max())
            assert float((got[i] - want).abs().max()) <= most * (4e-6 if dtype == torch.float32 else 2.0 ** -8), (splits, p)
