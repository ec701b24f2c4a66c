"""A retention state that two launches of one stream write one behind the other: a run step that goes on with an earlier run step's state, and
direct calls on one state.  Each must see what the launch before left, with overlapped launches as without them, to the bit."""

from dataclasses import replace

import pytest
import torch

import vobusun_models as M
from dryft_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_calls_in_a_row_on_one_state(dtype):
    H, d, dv, rot, n, calls = 16, 128, 128, 64, 4, 40
    gen = torch.Generator().manual_seed(1)
    projs = [(torch.randn(n, 2 * H * (d + dv), generator=gen) * 0.3).to(dtype).to(DEV) for _ in range(calls)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    inv = (100.0 ** (-torch.arange(rot // 2, dtype=torch.float64) * 2 / rot)).float().to(DEV)
    decay = torch.linspace(0.8, 0.99, H, dtype=torch.float64, device=DEV)
    slots, cu, pos = i32([3, 0, -1, 2]), i32(list(range(n + 1))), [i32([t, 2 * t, 0, t + 9]) for t in range(calls)]
    start = torch.randn(4, H, d, dv, generator=gen).to(DEV)

    def run(pdl):
        state, outs = start.clone(), [torch.zeros(n, H * dv, device=DEV, dtype=dtype) for _ in range(calls)]
        torch.cuda.synchronize()
        for t in range(calls):      # nothing but these launches in the stream
            K.retention_scan(projs[t], (0, H * d, 2 * H * d, 2 * H * d + H * dv), cu, slots, pos[t], inv, rot, decay, state, outs[t], n, H, d, dv,
                             d ** -0.5, 1e-6, one_token=True, pdl=pdl)
        return torch.stack(outs), state

    want, got = run(False), run(True)
    assert torch.isfinite(want[1]).all() and torch.equal(want[1][1], start[1])
    assert torch.equal(got[1], want[1]) and torch.equal(got[0], want[0])


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_a_borrowed_state_with_and_without_overlapped_launches(dtype):
    from dryft_b200.config import RunStep, config_from_dict
    from dryft_b200.engine.api import Engine

    cfg = config_from_dict(M.config([M.retention(heads=8, dim=128, vdim=128, rot_dims=64, ff=None) for _ in range(3)], width=256))

    class Borrowing:      # steps 1 and 2 go on with the state of step 0
        to_dict = staticmethod(cfg.to_dict)

        @staticmethod
        def model_spec():
            return replace(cfg.model_spec(), schedule=(RunStep(0), RunStep(1, cache_from=0), RunStep(2, cache_from=0)))

    logits = {}
    for pdl in (True, False):
        for graphs in (True, False):
            eng = Engine.from_config(Borrowing, seed=3, std=0.1, dtype=dtype, max_batch=4, max_seq_len=128, max_tokens=512, pdl=pdl, cuda_graphs=graphs)
            assert eng.cache.state(1) is eng.cache.state(0) and eng.cache.state(2) is eng.cache.state(0)
            with torch.inference_mode():
                slots = eng.cache.open_sequences(3)
                out = [eng.stepper.step(slots, [[1, 2, 3], [4] * 9, [5]], [[2], [8], [0]])]
                for t in range(12):
                    eng.cache.last_token.index_copy_(0, torch.tensor(slots, device=DEV), torch.tensor([t + 1, 2 * t, 3], dtype=torch.int32, device=DEV))
                    out.append(eng.stepper.decode_from_state(slots)[:3].clone())
            logits[pdl, graphs] = torch.cat(out)
    for key, got in logits.items():
        assert torch.isfinite(got).all() and torch.equal(got, logits[False, False]), key
