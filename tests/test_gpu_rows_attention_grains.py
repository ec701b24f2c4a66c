"""Row-wise attention whose splits are multiples of 16 keys: lengths and windows around the grains' and pages' edges, as many splits as
grains and more (empty ones write no values: what their buffers held must not matter), against 32-bit attention over the same keys."""

import math

import pytest
import torch

from test_gpu_kernels import DEV, K, _attn_ref, _fill_cache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_heads,n_kv,d", [(8, 2, 128), (16, 1, 32), (6, 2, 48)])
@pytest.mark.parametrize("window", [None, 70])
def test_splits_of_sixteen_keys(dtype, n_heads, n_kv, d, window):
    k = K()
    page, scale = 64, 1.0 / math.sqrt(d)
    positions = [0, 14, 15, 16, 31, 63, 64, 65, 130, 200, 519]
    n, g = len(positions), torch.Generator().manual_seed(d)
    seqs = {i: (torch.randn(p + 1, n_kv, d, generator=g).to(dtype), torch.randn(p + 1, n_kv, d, generator=g).to(dtype)) for i, p in enumerate(positions)}
    q = torch.randn(n + 1, n_heads, d, generator=g).to(dtype)
    kc, vc, pt = _fill_cache(seqs, n_kv, d, page, dtype, n_pages=40, max_pages=9, slots=n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    for splits in (1, 2, 5, 32, 130):
        out = torch.full((n + 1, n_heads * d), 9.0, device=DEV, dtype=dtype)
        po = torch.full((n + 1, n_heads, splits, d), float("nan"), device=DEV)
        pm = torch.full((n + 1, n_heads, splits, 2), float("nan"), device=DEV)
        k.attn_rows(q.to(DEV), kc, vc, pt, i32([*range(n), -1]), i32([*positions, 0]), out, scale, window, splits, po, pm)
        got = out.cpu().float()
        assert torch.count_nonzero(got[n]) == 0
        for i, p in enumerate(positions):
            want = _attn_ref(q[i], *seqs[i], p, scale, window)
            # 32-bit sums of up to 520 terms in other orders, then one rounding to the type of the result
            most = float(seqs[i][1].float().abs().max())
            assert float((got[i] - want).abs().max()) <= most * (2e-6 if dtype == torch.float32 else 2.0 ** -8), (splits, p)
