"""When a layer of experts multiplies grouped (each expert's weights read once) and when assignment by assignment."""

from types import SimpleNamespace

import pytest
import torch

from dryft_b200.parts.moe import MoE


def _layer(experts, top, hidden, inter, gated=True, tcgen05=True):
    layer = MoE.__new__(MoE)
    layer.rt = SimpleNamespace(tcgen05=tcgen05)
    layer.experts, layer.top, layer.hidden, layer.inter, layer.use_grouped = experts, top, hidden, inter, True
    layer.w_gate_up = torch.empty((experts, (2 if gated else 1) * inter, hidden), dtype=torch.bfloat16, device="meta")
    layer.w_down = torch.empty((experts, hidden, inter), dtype=torch.bfloat16, device="meta")
    layer._plan_grouped()
    return layer


@pytest.mark.parametrize("shape,first", [((64, 8, 2048, 768), 6), ((32, 4, 1024, 512), 15), ((8, 2, 64, 64), 32), ((64, 8, 2048, 760), 32), ((4, 4, 4096, 4096), 2),
                                         ((6144, 64, 4096, 4096), 3), ((6145, 64, 4096, 4096), 32)])
def test_grouped_from_the_tokens_that_spare_the_bytes(shape, first):
    """Below 32 tokens: where the weights spared reach 100 MB, and only where the tensor-core form takes the sizes."""
    layer = _layer(*shape)
    assert [n for n in range(1, 64) if layer._grouped(n)] == list(range(first, 64))


def test_switches():
    assert not _layer(64, 8, 2048, 768, tcgen05=False)._grouped(16) and _layer(64, 8, 2048, 768, tcgen05=False)._grouped(32)
    layer = _layer(64, 8, 2048, 768)
    layer.use_grouped = False
    assert not layer._grouped(16) and not layer._grouped(2048)
