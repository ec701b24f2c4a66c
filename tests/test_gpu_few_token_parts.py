"""Parts' kernels for steps of few tokens: matrices folded over the heads, the gates of a recurrence, joined splits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,heads,rows,cols", [(1, 16, 512, 128), (3, 2, 128, 512), (2, 3, 700, 200), (1, 1, 1, 1), (4, 2, 33, 77), (2, 2, 513, 132)])
def test_folded_matrices(dtype, n, heads, rows, cols):
    from dryft_b200.ops import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)
    w = randn(heads, rows, cols)
    q = randn(n, heads, rows + 5)
    out = torch.empty(heads, n, cols, device="cuda")
    K.latent_fold_q(q, w, out, rows)
    exact = torch.einsum("nhd,hdr->hnr", q[:, :, :rows].double(), w.double())
    scale = torch.einsum("nhd,hdr->hnr", q[:, :, :rows].double().abs(), w.double().abs())
    assert bool(((out.double() - exact).abs() <= (rows + 1) * 2.0 ** -24 * scale).all())
    o_lat, gate = randn(heads, n, rows), randn(n, 3 + heads * cols)
    for per_value in (False, True):
        y = torch.empty(n, heads * cols, dtype=dtype, device="cuda")
        K.latent_unfold_o(o_lat, w, gate, 3, y, per_value=per_value)
        g = torch.sigmoid(gate[:, 3:3 + heads * (cols if per_value else 1)].double()).view(n, heads, -1)
        e = torch.einsum("hnr,hrv->nhv", o_lat.double(), w.double()) * g
        s = torch.einsum("hnr,hrv->nhv", o_lat.double().abs(), w.double().abs()) * g
        unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24
        assert bool(((y.double().view(n, heads, cols) - e).abs() <= unit * e.abs() + (rows + 8) * 2.0 ** -23 * s).all())


@pytest.mark.parametrize("blocks,nb", [(2, 128), (3, 20), (1, 132), (4, 4), (2, 7)])
def test_recurrence_gates_of_few_and_many_tokens(blocks, nb):
    """A step of 70 tokens (the prompt form) against the same tokens in steps of 1 to 64 (the form for few), two sequences."""
    from dryft_b200.ops import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(nb)
    c, taps = blocks * nb, 4
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    proj, yb, xb, conv, cb = randn(70, 2 * c), randn(c) * 0.1, randn(c) * 0.1, randn(c, taps) * 0.5, randn(c) * 0.1
    wg, ba, bi, lam = randn(blocks, nb, 2, nb) * nb ** -0.5, randn(c), randn(c), torch.rand(c, generator=gen, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")

    def run(cuts):
        state, tail = torch.zeros(3, c, device="cuda"), torch.zeros(3, taps - 1, c, device="cuda")
        outs = [[], []]
        lens = [[n for n in cuts], [n for n in cuts]]
        at = [0, 35]
        for na, nb_ in zip(*lens):
            rows = torch.cat([proj[at[0]:at[0] + na], proj[at[1]:at[1] + nb_]]).contiguous()
            out = torch.empty(na + nb_, c, device="cuda")
            K.rglru(rows, 0, c, yb, xb, i32([0, na, na + nb_]), i32([2, 0]), i32([2] * na + [0] * nb_), conv, cb, wg, ba, bi, lam, 8.0, state, tail, out, 2, blocks)
            outs[0].append(out[:na])
            outs[1].append(out[na:])
            at = [at[0] + na, at[1] + nb_]
        return torch.cat(outs[0] + outs[1]), state

    whole, s0 = run([35])
    for cuts in ([1] * 35, [4, 31], [32, 3]):
        parts, s1 = run(cuts)
        torch.testing.assert_close(parts, whole, rtol=2e-5, atol=2e-5)      # sums of up to 132 products in two orders, carried over 35 steps
        torch.testing.assert_close(s1, s0, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("blocks,nb", [(2, 128), (3, 20), (1, 132), (4, 4), (2, 7), (1, 300)])
def test_recurrence_gates_do_not_depend_on_company(blocks, nb):
    """A sequence's token gives the same bits alone, in the form for few tokens and among so many that the prompt form takes it."""
    from dryft_b200.ops import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(nb)
    c, taps, seqs = blocks * nb, 4, 90
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    proj, yb, xb, conv, cb = randn(seqs, 2 * c), randn(c) * 0.1, randn(c) * 0.1, randn(c, taps) * 0.5, randn(c) * 0.1
    wg, ba, bi, lam = randn(blocks, nb, 2, nb) * nb ** -0.5, randn(c), randn(c), torch.rand(c, generator=gen, device="cuda")
    state0, tail0 = randn(seqs, c), randn(seqs, taps - 1, c)

    def run(who):
        n = len(who)
        at = torch.tensor(who, dtype=torch.int32, device="cuda")
        state, tail, out = state0.clone(), tail0.clone(), torch.empty(n, c, device="cuda")
        cu = torch.arange(n + 1, dtype=torch.int32, device="cuda")
        K.rglru(proj[who].contiguous(), 0, c, yb, xb, cu, at, at, conv, cb, wg, ba, bi, lam, 8.0, state, tail, out, n, blocks)
        return out, state[who]

    everyone = list(range(seqs))
    out, state = run(everyone)
    for who in ([0], [7, 3], everyone[10:19], everyone[20:84], everyone[25:90]):
        o, s = run(who)
        assert torch.equal(o, out[who]) and torch.equal(s, state[who]), len(who)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,rows,cols", [(2, 64, 256), (4, 65, 132), (3, 128, 512), (2, 513, 77), (16, 512, 128), (1, 300, 40), (5, 1030, 24)])
def test_folded_matrices_do_not_depend_on_company(dtype, heads, rows, cols):
    """A token's fold has the same bits alone, where threads share a column, and among so many that a thread takes whole columns."""
    from dryft_b200.ops import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)
    n = 700
    w, q, o_lat, gate = randn(heads, rows, cols), randn(n, heads, rows + 5), randn(heads, n, rows), randn(n, heads)

    def run(who):
        lat, out = torch.empty(heads, len(who), cols, device="cuda"), torch.empty(len(who), heads * cols, dtype=dtype, device="cuda")
        K.latent_fold_q(q[who].contiguous(), w, lat, rows)
        K.latent_unfold_o(o_lat[:, who].contiguous(), w, gate[who].contiguous(), 0, out)
        return lat, out

    lat, out = run(list(range(n)))
    exact, scale = (torch.einsum("nhd,hdr->hnr", a[:, :, :rows].double(), b.double()) for a, b in ((q, w), (q.abs(), w.abs())))
    assert bool(((lat.double() - exact).abs() <= (rows + 1) * 2.0 ** -24 * scale).all())
    for who in ([0], [699], [5, 600], list(range(40, 49)), list(range(100, 164))):
        a, b = run(who)
        assert torch.equal(a, lat[:, who]) and torch.equal(b, out[who]), len(who)
