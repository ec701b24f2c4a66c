"""Retention of steps in which every sequence brings one token: the kernel of their own against the plain recurrence in 64-bit, at widths
that fill and that do not fill its 16-byte words and row groups (values of 300 leave threads over, 24 of 64 dims two rows a thread), with
padding sequences, and at widths that it leaves to the walk."""

import pytest
import torch

from test_gpu_kernels import DEV
from test_gpu_vobusun_parts import _retention_plain
from dryft_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H, d, dv, rot", [(2, 16, 24, 8), (16, 128, 128, 128), (3, 64, 24, 64), (2, 12, 300, 4), (1, 7, 4, 0), (1, 9, 6, 2), (1, 300, 128, 300)])
def test_steps_of_one_token(dtype, H, d, dv, rot):
    T, base, eps, slots = 6, 1000.0, 1e-6, 4
    gen = torch.Generator().manual_seed(d + dv)
    decay = [0.97 - 0.1 * (h % 4) for h in range(H)]
    new = lambda w: (torch.randn(3, T, H, w, generator=gen) * 0.5).to(dtype)
    q, k, v, g = new(d), new(d), new(dv), new(dv)
    want = torch.stack([_retention_plain(*(t[s].double() for t in (q, k, v, g)), decay, rot, base, eps) for s in range(3)])
    state = torch.zeros(slots, H, d, dv, device=DEV)
    state[0] = 7.0                                        # nobody's: a padding sequence must leave it alone
    inv = (base ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / max(rot, 1))).float().to(DEV)
    dec = torch.tensor(decay, dtype=torch.float64, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    where, offs = [2, -1, 1, 3], (0, H * d, 2 * H * d, 2 * H * d + H * dv)
    for t in range(T):
        rows = torch.cat([x[:, t].reshape(3, -1) for x in (q, k, v, g)], dim=1)
        proj = torch.stack([rows[0], torch.full_like(rows[0], float("nan")), rows[1], rows[2]]).to(DEV)
        out = torch.zeros(4, H * dv, device=DEV, dtype=dtype)
        K.retention_scan(proj, offs, i32(list(range(5))), i32(where), i32([t, 0, t, t]), inv, rot, dec, state, out, 4, H, d, dv, d ** -0.5, eps,
                         one_token=True, pdl=bool(t & 1))
        got = out.double().cpu()[[0, 2, 3]]
        # 32-bit states and sums of up to 300 terms, a norm over them; one rounding of the result
        bound = (4e-6 if dtype == torch.float32 else 2.0 ** -8) * float(want[:, t].abs().max()) + 1e-6
        assert float((got - want[:, t]).abs().max()) <= bound, t
    assert torch.all(state[0] == 7.0)
    with pytest.raises(K.KernelError):
        K.retention_scan(proj, offs, i32([0, 4]), i32([1]), i32([0] * 4), inv, rot, dec, state, out, 1, H, d, dv, 1.0, eps, one_token=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H, d, dv, rot", [(2, 32, 128, 16), (1, 33, 128, 0), (2, 64, 128, 64), (1, 65, 128, 2)])
def test_rows_a_thread_around_those_that_have_a_kernel(dtype, H, d, dv, rot):
    """Four, five, eight and nine rows a thread."""
    test_steps_of_one_token(dtype, H, d, dv, rot)
