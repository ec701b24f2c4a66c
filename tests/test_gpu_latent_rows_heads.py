"""Row-wise latent attention with two and with four heads a warp (few and many blocks): a token's result has the same bits either way, with
splits that have no keys, ranks that are no multiple of four and heads that do not exist."""

import pytest
import torch

from test_gpu_kernels import DEV
from test_gpu_vobusun_parts import i32
from dryft_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kv_rank, rot, H, n_splits", [(40, 16, 3, 1), (40, 16, 18, 5), (70, 2, 9, 33), (17, 0, 8, 2), (512, 64, 16, 40)])
def test_few_and_many_blocks(dtype, kv_rank, rot, H, n_splits):
    torch.manual_seed(kv_rank)
    page, n = 64, 160                                   # 160 blocks at least: four heads a warp; a token alone: two
    k_pages = torch.randn(4, 1, page, kv_rank + rot, device=DEV).to(dtype)
    table = i32([[0, 0, 0, 0], [2, 0, 3, 1]])
    inv = torch.tensor([50.0 ** (-2.0 * j / rot) for j in range(rot // 2)], dtype=torch.float32, device=DEV) if rot else None
    q_lat = torch.randn(H, n, kv_rank, device=DEV) * 0.3
    q = torch.randn(n, H, 5 + rot, device=DEV).to(dtype)
    pos = torch.randint(0, 4 * page, (n,)).tolist()
    pos[:4] = [0, 31, 32, 255]

    def rows(of):
        out = torch.full((H, len(of), kv_rank), float("nan"), device=DEV, dtype=dtype)
        K.latent_attn_rows(q_lat[:, of].contiguous(), q[of].contiguous(), 5, k_pages, table, i32([1] * len(of)), i32([pos[t] for t in of]), inv, True,
                           out, kv_rank, rot, 0.2, 100, n_splits=n_splits)
        return out

    together = rows(list(range(n)))
    assert torch.isfinite(together).all()
    for t in (0, 1, 2, 3, 4, 77, 159):
        assert torch.equal(rows([t])[:, 0], together[:, t]), t


def test_more_heads_than_a_grid_has_rows():
    """65,537 heads in blocks of 16: the first, the last and some between against one head alone."""
    torch.manual_seed(3)
    kv_rank, H = 16, 65537
    k_pages, table = torch.randn(1, 1, 64, kv_rank, device=DEV), i32([[0]])
    q_lat, q = torch.randn(H, 1, kv_rank, device=DEV), torch.zeros(1, H, 1, device=DEV)

    def rows(heads):
        out = torch.full((len(heads), 1, kv_rank), float("nan"), device=DEV)
        K.latent_attn_rows(q_lat[heads].contiguous(), q[:, heads].contiguous(), 1, k_pages, table, i32([0]), i32([40]), None, True, out, kv_rank, 0, 0.2, None)
        return out

    together = rows(list(range(H)))
    for h in (0, 15, 16, 32767, 65535, 65536):
        assert torch.equal(rows([h])[0], together[h]), h
