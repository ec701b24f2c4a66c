"""The engine's switch for overlapped launches (``pdl``) reaches every kernel: a captured step holds programmatic edges with it and
none without, and the results are the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def programmatic_edges(fn) -> int:
    """Edges of a captured ``fn()`` on which a launch may start before the one in front of it has ended (nothing is run)."""
    from cuda.bindings import runtime as R

    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        keep = fn()
    rc, _, _, data, n = R.cudaGraphGetEdges_v2(R.cudaGraph_t(graph.raw_cuda_graph()), 20000)
    assert rc == R.cudaError_t.cudaSuccess and 0 < n < 20000, rc
    del keep
    return sum(int(e.type) == int(R.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic) for e in data[:n])


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("name", ["tiny-256", "tevovik-tiny", "vobusun-tiny", "mogelix-tiny", "kerirax-tiny", "dusupel-tiny", "puturax-tiny"])
def test_a_step_without_overlap_has_none_and_gives_the_same_bits(name, dtype):
    from dryft_b200.config import preset
    from dryft_b200.engine.api import Engine

    cfg = dict(preset("tiny-b"), hidden_size=256, head_dim=64) if name == "tiny-256" else preset(name)
    logits = {}
    for pdl in (True, False):
        for graphs in (True, False):
            eng = Engine.from_config(cfg, seed=3, dtype=dtype, max_batch=8, max_seq_len=256, max_tokens=1024, pdl=pdl, cuda_graphs=graphs)
            with torch.inference_mode():
                slots = eng.cache.open_sequences(3)
                out = [eng.stepper.step(slots, [[1, 2, 3], [4] * 9, [5]], [[2], [8], [0]])]
                for t in range(6):
                    eng.cache.last_token.index_copy_(0, torch.tensor(slots, device="cuda"), torch.tensor([t + 1, 2 * t, 3], dtype=torch.int32, device="cuda"))
                    out.append(eng.stepper.decode_from_state(slots)[:3].clone())
                if graphs:
                    (g,) = eng.stepper._graphs.values()
                    g.seq_slot.fill_(-1)                     # padding only: the run in front of the capture changes nothing
                    n = programmatic_edges(g._body)
                    assert n == 0 if not pdl else n > 0 or dtype == "float32", (n, pdl)      # 32-bit products up to 256 wide have no such form
            logits[pdl, graphs] = torch.cat(out)
    for key, got in logits.items():
        assert torch.isfinite(got).all() and torch.equal(got, logits[True, True]), key


def test_experts_products_follow_the_switches():
    from dryft_b200.ops import kernels as K

    n, e, width, f, top = 40, 8, 128, 64, 2
    h = torch.randn(n, width, device="cuda").bfloat16()
    w1, w2 = (torch.randn(e, 2 * f, width, device="cuda") * 0.1).bfloat16(), (torch.randn(e, width, f, device="cuda") * 0.1).bfloat16()
    idx = torch.stack([torch.randperm(e, device="cuda")[:top] for _ in range(n)]).to(torch.int32)
    out = {}
    for pdl in (True, False):
        for tc in (True, False):
            out[pdl, tc] = torch.empty(n * top, width, dtype=torch.bfloat16, device="cuda")
            edges = programmatic_edges(lambda: K.moe_grouped(h, w1, w2, idx, out[pdl, tc], pdl=pdl, tcgen05=tc))
            assert edges == (2 if pdl and tc else 0), (pdl, tc, edges)
    assert torch.equal(out[True, True], out[False, True]) and torch.equal(out[True, False], out[False, False])
    exact = out[True, False].double()
    assert float((out[True, True].double() - exact).norm() / exact.norm()) < 4.0 * 2.0 ** -8      # two roundings on either side
    K.check_error_flags()
