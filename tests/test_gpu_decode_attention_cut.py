"""Decode attention of one launch whose rows end on both sides of the length up to which a cluster's first block works alone: rows of 1
key to four pages and a little more, in clusters of 2, 6 and 8, against 32-bit attention over the same keys."""

import math

import pytest
import torch

from test_gpu_kernels import DEV, K, _attn_ref, _fill_cache

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.mark.parametrize("n_heads,n_kv,d", [(8, 2, 128), (16, 1, 32), (2, 2, 64), (6, 2, 48)])
@pytest.mark.parametrize("window", [None, 250])
def test_rows_around_the_cut(n_heads, n_kv, d, window):
    k = K()
    page, scale = 64, 1.0 / math.sqrt(d)
    lengths = [0, 1, 15, 16, 127, 128, 254, 255, 256, 257, 270, 320, 513]      # cached keys; the new token's own is one more
    n, g = len(lengths), torch.Generator().manual_seed(d)
    seqs, rows = {}, []
    for i, length in enumerate(lengths):
        kseq, vseq = torch.randn(length + 1, n_kv, d, generator=g).to(BF), torch.randn(length + 1, n_kv, d, generator=g).to(BF)
        q = torch.randn(n_heads, d, generator=g).to(BF)
        rows.append(torch.cat([q.reshape(-1), kseq[length].reshape(-1), vseq[length].reshape(-1)]))
        seqs[i] = (kseq, vseq)
    qkv = torch.stack(rows + rows[:1])          # the last row is padding
    want = [_attn_ref(qkv[i, :n_heads * d].view(n_heads, d), *seqs[i], lengths[i], scale, window) for i in range(n)]
    for splits in (2, 6, 8):
        kc, vc, pt = _fill_cache(seqs, n_kv, d, page, BF, n_pages=60, max_pages=9, slots=n, scatter_seed=splits)
        for i, length in enumerate(lengths):      # the launch itself writes the new token's row; what lies there and behind is NaN
            for c in (kc, vc):
                c[int(pt[i, length // page]), :, length % page:] = float("nan")
        out = torch.full((n + 1, n_heads * d), 9.0, device=DEV, dtype=BF)
        k.attn_decode(qkv.to(DEV), None, None, None, torch.tensor([*range(n), -1], dtype=torch.int32, device=DEV),
                      torch.tensor([*lengths, 0], dtype=torch.int32, device=DEV), kc, vc, pt, out, n_heads, n_kv, d, 0, 0.0, scale, window, splits)
        got = out.cpu().float()
        assert torch.count_nonzero(got[n]) == 0
        for i, length in enumerate(lengths):
            # probabilities are rounded to bfloat16 before they meet the values (2^-9 of each, so 2^-9 of the largest value), the result
            # once (2^-9 of it), and the new key and value not at all; a half more for the 32-bit sums and exponentials
            bound = 1.5 * 2.0 ** -8 * float(seqs[i][1].float().abs().max())
            assert float((got[i] - want[i]).abs().max()) <= bound, (splits, length)
            assert torch.equal(kc[int(pt[i, length // page]), :, length % page].cpu(), seqs[i][0][length]), (splits, length)
