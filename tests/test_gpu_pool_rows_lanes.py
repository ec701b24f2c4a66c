"""Row-wise attention over pages with one lane a key (many rows) and with two (few): the same rows in both forms against 64-bit, at
key counts around the tiles of either."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D,DV,group", [(192, 128, 1), (128, 128, 4), (24, 24, 1), (16, 16, 2)])
@pytest.mark.parametrize("splits,mods", [(1, False), (3, False), (1, True)])
def test_few_and_many_rows_attend_alike(D, DV, group, splits, mods, dtype):
    from dryft_b200.ops import kernels as K

    G, page, H = 2, 64, 2 * group
    gen = torch.Generator("cuda").manual_seed(D + DV + splits)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    lens = [1, 2, 15, 16, 17, 31, 32, 33, 47, 64, 65, 129, 200, 300]
    keys = max(lens)
    n_pages = (keys + page - 1) // page
    kp, vp = rnd(n_pages + 1, G, page, D).to(dtype), rnd(n_pages + 1, G, page, DV).to(dtype)
    table = torch.randperm(n_pages, generator=torch.Generator().manual_seed(3)).int().cuda()[None] + 1
    kp[0] = vp[0] = float("nan")                    # no sequence's page
    q = rnd(len(lens), H, D).to(dtype)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda")
    kw = dict(softcap=3.0, dist_bias=(rnd(H).abs(), rnd(H).abs())) if mods else {}

    def run(rep):                                   # `rep` copies of every row: beyond 444 blocks the one-lane form
        n = len(lens) * rep
        slot = torch.zeros(n, dtype=torch.int32, device="cuda")
        po, pm = torch.full((n, H, splits, DV), float("nan"), device="cuda"), torch.full((n, H, splits, 2), float("nan"), device="cuda")
        out = torch.full((n, H, DV), float("nan"), device="cuda", dtype=dtype)
        K.pool_attn_rows(q.repeat(rep, 1, 1), kp, vp, table, None, None, slot, pos.repeat(rep), out, 0.2, 1 << 30, 0, splits, po, pm, **kw)
        return out[-len(lens):].double()

    few, many = run(1), run(40)
    kk, vv = (t[table[0].long()].double().permute(1, 0, 2, 3).flatten(1, 2) for t in (kp, vp))      # [G, keys, size]
    for i, n in enumerate(lens):
        for h in range(H):
            s = 0.2 * (kk[h // group, :n] @ q[i, h].double())
            if mods:
                r1, r2 = (t[h].double() for t in kw["dist_bias"])
                s = 3.0 * torch.tanh(s / 3.0) - r1 * torch.log1p(r2 * torch.arange(n - 1, -1, -1, device="cuda").double())
            want = torch.softmax(s, 0) @ vv[h // group, :n]
            # values of spread one: 32-bit sums over at most 300 keys, and for bfloat16 one rounding of the result (2^-9 of it)
            tol = dict(rtol=2.0 ** -8, atol=1e-4) if dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)
            torch.testing.assert_close(few[i, h], want, **tol)
            torch.testing.assert_close(many[i, h], want, **tol)
