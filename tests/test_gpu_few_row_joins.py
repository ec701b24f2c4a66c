"""Joins, layer norms and activations of few rows, whose launches overlap the launch before them, on both sides of the row and width
limits of that form."""

import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 1e-5


def _bound(dtype):      # one rounding to the output's type (bfloat16: 2^-9 relative), or 32-bit sums of a few thousand terms
    return dict(rtol=2.0 ** -8, atol=2.0 ** -9) if dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)


def _chain(n, width, streams, dtype, steps, sync):
    """``steps`` products, activations, joins and layer norms that read one another's results, launched one behind the other."""
    from dryft_b200.ops import kernels as K

    g = torch.Generator("cuda").manual_seed(7 * n + width + streams)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x = rnd(n, streams, width)
    mix = torch.eye(streams, device="cuda") * 0.7 + 0.05 * rnd(streams, streams)
    outw, inw, w, b = rnd(streams), rnd(streams), 1 + 0.1 * rnd(width), 0.1 * rnd(width)
    gu = rnd(n, 2 * width).to(dtype)
    y, h, h2 = (torch.empty(n, width, device="cuda", dtype=dtype) for _ in range(3))
    x32 = rnd(n, width)
    ref = [t.double() for t in (x, gu, x32)]
    for _ in range(steps):
        K.glu_clamp(gu, y, 0.9, 1.3, 0.5)
        if sync: torch.cuda.synchronize()
        K.hc_step(x, streams, x_out=x, y=y, mix=mix, outw=outw, mult=0.6, inw=inw, norm_w=w, eps=EPS, h=h)
        if sync: torch.cuda.synchronize()
        K.stream_sum_ln(x32, [(h, 0.5), (y, 0.25)], norms=[(w, b, h2)], eps=EPS)
        if sync: torch.cuda.synchronize()
        gu[:, :width].copy_(h2)
    return ref, (mix, outw, inw, w, b), (x, y, h, x32, h2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("streams", [1, 3, 4, 8])
@pytest.mark.parametrize("n,width", [(1, 2048), (16, 1028), (17, 1024), (16, 1030), (2, 36), (3, 4100), (40, 2048)])
def test_joins_against_64_bits_and_launched_one_behind_the_other(n, width, streams, dtype):
    (x, gu, x32), (mix, outw, inw, w, b), got = _chain(n, width, streams, dtype, 1, False)
    gate, up = gu[:, :width].clamp(max=0.9), gu[:, width:].clamp(-0.9, 0.9)
    y = gate * torch.sigmoid(1.3 * gate) * (up + 0.5)
    torch.testing.assert_close(got[1].double(), y, **_bound(dtype))
    y = got[1].double()
    x = torch.einsum("st,nsw->ntw", mix.double(), x) + 0.6 * outw.double()[None, :, None] * y[:, None]
    torch.testing.assert_close(got[0].double(), x, rtol=2e-5, atol=2e-5)
    u = torch.einsum("t,ntw->nw", inw.double(), x)
    torch.testing.assert_close(got[2].double(), u / (u.square().mean(1, keepdim=True) + EPS).sqrt() * w.double(), **_bound(dtype))
    z = x32 + 0.5 * got[2].double() + 0.25 * y
    torch.testing.assert_close(got[3].double(), z, rtol=2e-5, atol=2e-5)
    torch.testing.assert_close(got[4].double(), torch.nn.functional.layer_norm(z, (width,), w.double(), b.double(), EPS), **_bound(dtype))
    # many steps without a stop in between leave the bits of the same steps with the device idle before each launch
    for a, c in zip(_chain(n, width, streams, dtype, 12, False)[2], _chain(n, width, streams, dtype, 12, True)[2]):
        assert torch.isfinite(a).all() and torch.equal(a, c)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("streams", [1, 2, 4, 8])
@pytest.mark.parametrize("width", [36, 1022, 1024, 1028, 1030, 2048, 2050, 4100])
def test_joins_do_not_depend_on_company(width, streams, dtype):
    """A row's join, layer norms and activation have the same bits among few rows and among many, whose blocks have half the threads."""
    from dryft_b200.ops import kernels as K

    g = torch.Generator("cuda").manual_seed(width + streams)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    n = 40
    x, mix, outw, inw, w, b = rnd(n, streams, width), rnd(streams, streams), rnd(streams), rnd(streams), 1 + 0.1 * rnd(width), 0.1 * rnd(width)
    y, gu, x32 = rnd(n, width).to(dtype), rnd(n, 2 * width).to(dtype), rnd(n, width)

    def run(rows):
        xs, ys, x32s = x[rows].contiguous(), y[rows].contiguous(), x32[rows].contiguous()
        h, h1, h2, act = (torch.empty(len(rows), width, device="cuda", dtype=dtype) for _ in range(4))
        K.hc_step(xs, streams, x_out=xs, y=ys, mix=mix, outw=outw, mult=0.6, inw=inw, norm_w=w, eps=EPS, h=h)
        K.stream_sum_ln(x32s, [(h, 0.5), (ys, 0.25), (h, -1.0)], norms=[(w, b, h1), (b, w, h2)], eps=EPS)
        K.glu_clamp(gu[rows].contiguous(), act, 0.9, 1.3, 0.5)
        return xs, h, x32s, h1, h2, act

    many = run(list(range(n)))
    for rows in ([0], [39, 3], list(range(16)), list(range(20, 37))):
        for a, c in zip(run(rows), many):
            assert torch.isfinite(a).all() and torch.equal(a, c[rows]), len(rows)
