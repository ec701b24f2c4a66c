"""Decode attention of one launch with per-head norms and rotation, against plain attention over the same keys: the new token's key and value
are cached as the plain parts make them, and nothing else in the cache is written, whichever way a row's keys are split over blocks."""

import math

import pytest
import torch

import plain_qwen3 as P
from test_gpu_kernels import ATTN_BF16_TOL, DEV, K, _attn_ref, _fill_cache

pytestmark = pytest.mark.gpu

BF = torch.bfloat16
# (splits, block shape, splits combined inside a thread-block cluster or through memory)
WAYS = ((1, -1, True), (1, 0, True), (2, 0, True), (3, -1, True), (6, -1, True), (8, 2, True), (7, 1, True), (3, -1, False), (7, 0, False),
        (12, -1, True))


def _check(n_heads, n_kv, d, rot, window, cached, ways, padding_pos):
    """Rows that go on after ``cached[i]`` tokens, and two padding rows, one of them at position ``padding_pos``."""
    k, g = K(), torch.Generator().manual_seed(d + n_heads)
    page, theta, eps, scale = 64, 1e4, 1e-5, 1.0 / math.sqrt(d)
    n, slots, pos = len(cached) + 2, [-1, *range(len(cached)), -1], [padding_pos, *cached, 0]
    old = {i: (torch.randn(c, n_kv, d, generator=g).to(BF), torch.randn(c, n_kv, d, generator=g).to(BF)) for i, c in enumerate(cached)}
    qkv = torch.randn(n, (n_heads + 2 * n_kv) * d, generator=g).to(BF)
    wq, wk = ((1 + 0.1 * torch.randn(d, generator=g)).to(BF).float() for _ in range(2))
    inv_freq = 1.0 / (theta ** (torch.arange(0, rot, 2, dtype=torch.int64).float() / rot))
    cos, sin = P.rope_cos_sin(torch.tensor(pos), rot, theta, BF)
    turned = lambda x: torch.cat((P.apply_rope(x[..., :rot], cos, sin), x[..., rot:]), dim=-1)
    q, kn, vn = qkv.view(n, -1, d).split([n_heads, n_kv, n_kv], dim=1)
    q, kn = turned(P.rmsnorm(q, wq, eps)), turned(P.rmsnorm(kn, wk, eps))
    want = torch.zeros(n, n_heads * d)
    for r, s in enumerate(slots):
        if s >= 0:
            want[r] = _attn_ref(q[r], torch.cat([old[s][0], kn[r][None]]), torch.cat([old[s][1], vn[r][None]]), pos[r], scale, window, p_round=BF)
    room = lambda x: torch.cat([x, torch.full((1, n_kv, d), 55.0, dtype=BF)])      # pages for one token more than are cached
    n_pages = sum(c // page + 1 for c in cached) + 2
    for splits, shape, cluster in ways:
        what = f"splits {splits}, shape {shape}, cluster {cluster}"
        kc, vc, pt = _fill_cache({s: (room(a), room(b)) for s, (a, b) in old.items()}, n_kv, d, page, BF, n_pages=n_pages,
                                 max_pages=max(cached) // page + 1, slots=len(cached), scatter_seed=splits)
        kc0, vc0 = kc.clone(), vc.clone()
        out = torch.full((n, n_heads * d), 9.0, device=DEV, dtype=BF)
        po, pm = torch.empty(n, n_heads, splits, d, device=DEV), torch.empty(n, n_heads, splits, 2, device=DEV)
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        k.attn_decode(qkv.to(DEV), wq.to(DEV), wk.to(DEV), inv_freq.to(DEV), i32(slots), i32(pos), kc, vc, pt, out, n_heads, n_kv, d, rot, eps,
                      scale, window, splits, po, pm, shape=shape, cluster=cluster)
        torch.testing.assert_close(out.cpu().float(), want, **ATTN_BF16_TOL, msg=lambda m: f"{what}: {m}")
        assert torch.count_nonzero(out[0]) == 0 and torch.count_nonzero(out[-1]) == 0, what
        for c, c0, new in ((kc, kc0, kn), (vc, vc0, vn)):
            assert int((c != c0).any(dim=-1).sum()) == len(cached) * n_kv, what      # one row per live token and kv head
            for r, s in enumerate(slots):
                if s >= 0:
                    got = c[int(pt[s, pos[r] // page]), :, pos[r] % page].cpu()
                    torch.testing.assert_close(got.float(), new[r].float(), rtol=2e-2, atol=2e-2, msg=lambda m: f"{what}: {m}")


@pytest.mark.parametrize("n_heads,n_kv,d", [(8, 2, 208), (16, 1, 208), (4, 2, 192), (4, 2, 224)])
def test_head_sizes_whose_widest_block_is_near_the_shared_memory_limit(n_heads, n_kv, d):
    """A block of eight warps takes 220 KB at 208 dims: what blocks of a cluster receive does not fit beside it, everything else does."""
    ways = [w for w in WAYS if d < 224 or w[1] != 0]      # (eight warps of 224 dims fit no launch)
    _check(n_heads, n_kv, d, 64, None, [0, 63, 200, 300, 513], ways, 0)


@pytest.mark.parametrize("n_heads,n_kv,d,rot", [(8, 2, 128, 128), (4, 4, 64, 32), (12, 4, 96, 96), (16, 1, 32, 16), (4, 1, 256, 128)])
@pytest.mark.parametrize("window", [None, 300])
def test_rows_beyond_the_length_of_one_block(n_heads, n_kv, d, rot, window):
    """Rows on both sides of the lengths up to which a cluster's first block works alone (256 keys with eight warps, 192 and 96 with four and
    two), the new token in the last split's page and in the first, and padding whose position is far beyond them."""
    ways = [w for w in WAYS if d < 224 or w[1] != 0]
    _check(n_heads, n_kv, d, rot, window, [0, 40, 127, 190, 191, 192, 255, 256, 320, 513, 700], ways, 700)
