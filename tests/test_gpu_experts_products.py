"""The experts' products at the edges of their kernels: experts with no rows, one row, and row counts around 16, a tile and its
halves; inner sizes that do and do not fill a feature tile; every activation; few tokens that share experts."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(h, w1, w2, idx, act, in_w, limit, alpha, off):
    n, top = idx.shape
    f = w2.shape[2]
    y = torch.zeros(n, top, w2.shape[1], dtype=torch.float64, device=h.device)
    for e in range(w1.shape[0]):
        t, k = torch.nonzero(idx == e, as_tuple=True)
        if not len(t):
            continue
        z = h[t].double() @ w1[e].double().T
        if act == "relu2":
            a = z.clamp(min=0.0) ** 2
        else:
            g, u = z[:, :f], z[:, f:]
            if act == "clamped":
                s = in_w[t, k].double()[:, None]
                g, u = (g * s).clamp(max=limit), (u * s).clamp(-limit, limit)
                a = g * torch.sigmoid(alpha * g) * (u + off)
            else:
                a = g * torch.sigmoid(g) * u
        y[t, k] = a @ w2[e].double().T
    return y.reshape(n * top, -1)


def _case(n, top, e, width, f, act, rows=None, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed + 7 * n + width + f)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    h = randn(n, width).bfloat16()
    w1 = (randn(e, f if act == "relu2" else 2 * f, width) * width ** -0.5).bfloat16()
    w2 = (randn(e, width, f) * f ** -0.5).bfloat16()
    if rows is None:
        idx = torch.argsort(torch.rand(n, e, generator=gen, device="cuda"), dim=1)[:, :top].to(torch.int32).contiguous()
    else:      # expert i is chosen rows[i] times, in a mixed order (top == 1)
        idx = torch.repeat_interleave(torch.arange(len(rows), device="cuda"), torch.tensor(rows, device="cuda"))
        idx = idx[torch.randperm(len(idx), generator=gen, device="cuda")].to(torch.int32)[:, None].contiguous()
    in_w = torch.rand(idx.shape, generator=gen, device="cuda") + 0.2
    return h, w1, w2, idx, in_w


def _check(y, exact):
    # two bfloat16 roundings on the way (the activation, the result), each half a unit in 2^8 of its value
    err = (y.double() - exact).norm() / exact.norm()
    assert float(err) < 2.0 * 2.0 ** -8, float(err)
    assert float((y.double() - exact).abs().max()) < 2.0 ** -5 * float(exact.abs().max())


ROWS = [0, 1, 15, 16, 17, 0, 64, 65, 127, 128, 129, 200, 255, 256, 257, 3]


@pytest.mark.parametrize("act", ["silu", "relu2", "clamped"])
@pytest.mark.parametrize("width,f,rows", [
    (128, 64, ROWS),                                   # many rows of a few small experts: mma.sync
    (64, 192, ROWS),                                   # one k slice, a feature tile and a half
    (192, 320, [r * 6 for r in ROWS]),                 # tiles of 256 rows
    (256, 128, [700, 0, 1, 513]),
    (256, 64, ROWS), (128, 64, [128, 0, 1, 129, 255, 64]),   # less than a feature tile on tcgen05: not all too small, not too many rows
    (48, 80, ROWS), (112, 64, [r * 2 for r in ROWS]),  # inner sizes that the mma.sync products take
])
def test_grouped_products(act, width, f, rows):
    from dryft_b200.ops import kernels as K

    h, w1, w2, idx, in_w = _case(sum(rows), 1, len(rows), width, f, act, rows)
    y = torch.full((idx.numel(), width), float("nan"), dtype=torch.bfloat16, device="cuda")
    K.moe_grouped(h, w1, w2, idx, y, gated=act != "relu2", in_w=in_w if act == "clamped" else None, limit=1.5, alpha=1.702, up_offset=1.0)
    _check(y, _exact(h, w1, w2, idx, act, in_w, 1.5, 1.702, 1.0))
    K.check_error_flags()


def test_grouped_products_of_many_assignments():
    from dryft_b200.ops import kernels as K

    # more assignments than the sorting block keeps in registers, more experts than it has tables for every warp
    h, w1, w2, idx, in_w = _case(5000, 4, 500, 64, 64, "silu")
    y = torch.empty((idx.numel(), 64), dtype=torch.bfloat16, device="cuda")
    K.moe_grouped(h, w1, w2, idx, y)
    _check(y, _exact(h, w1, w2, idx, "silu", in_w, 0, 0, 0))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,top,e,width,f", [(1, 1, 1, 64, 24), (5, 3, 7, 128, 33), (16, 8, 24, 256, 72), (32, 8, 9, 64, 40), (4, 2, 64, 72, 16)])
def test_few_tokens_that_share_experts(dtype, n, top, e, width, f):
    """Assignment by assignment: an assignment among others has the bits that it has alone, whoever shares its expert."""
    from dryft_b200.ops import kernels as K

    h, w1, _, idx, in_w = _case(n, top, e, width, f, "silu")
    h, w1 = h.to(dtype), w1.to(dtype)
    for mode, w in (("gate_up", w1), ("down", w1), ("up_relu2", w1), ("gate_up_clamp", w1)):
        outs = w.shape[1] // 2 if mode.startswith("gate") else w.shape[1]
        kw = dict(in_w=in_w, limit=1.5, alpha=1.702, up_offset=1.0) if mode == "gate_up_clamp" else {}
        x = h if mode != "down" else torch.randn(n * top, width, device="cuda").to(dtype)
        out = torch.full((n * top, outs), float("nan"), dtype=dtype, device="cuda")
        K.moe_rows(x, w, idx, out, mode, **kw)
        for t in range(0, n, 3):
            alone = torch.empty((top, outs), dtype=dtype, device="cuda")
            if kw:
                kw["in_w"] = in_w[t:t + 1].contiguous()
            K.moe_rows(x[t:t + 1] if mode != "down" else x[t * top:(t + 1) * top], w, idx[t:t + 1].contiguous(), alone, mode, **kw)
            assert torch.equal(alone, out[t * top:(t + 1) * top]), mode


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,top,width", [(1, 1, 1), (3, 8, 64), (7, 9, 1000), (2, 17, 2056), (5, 2, 77)])
def test_weighted_sum(dtype, n, top, width):
    from dryft_b200.ops import kernels as K

    y, wts = torch.randn(n * top, width, device="cuda").to(dtype), torch.rand(n, top, device="cuda")
    out = torch.empty(n, width, dtype=dtype, device="cuda")
    K.moe_combine(y, wts, out)
    exact = (y.double().view(n, top, width) * wts.double()[..., None]).sum(1)
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    bound = unit * exact.abs() + 2.0 ** -23 * top * (y.double().view(n, top, width).abs() * wts.double()[..., None]).sum(1)
    assert bool(((out.double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("act", ["silu", "clamped"])
@pytest.mark.parametrize("n", [8, 300])
def test_activation_of_gates_far_below_zero(act, n):
    """Gates of -86 to -88.5: one plus the exponential is beyond 2^126, where a fast division gives zero.  With an up value of
    2^100 the activation is an ordinary bfloat16 number."""
    from dryft_b200.ops import kernels as K

    f = width = 64
    gates = torch.linspace(-88.5, -86.0, 6, device="cuda").repeat(11)[:f]          # steps of a half: exact in bfloat16
    w1 = torch.zeros(1, 2 * f, width, device="cuda")
    w1[0, :f, 0], w1[0, f:, 0] = gates, 2.0 ** 100
    w1, w2 = w1.bfloat16(), torch.eye(f, device="cuda")[None].bfloat16().contiguous()
    h = torch.zeros(n, width, dtype=torch.bfloat16, device="cuda")
    h[:, 0] = 1.0
    idx, in_w = torch.zeros(n, 1, dtype=torch.int32, device="cuda"), torch.ones(n, 1, device="cuda")
    y = torch.empty(n, width, dtype=torch.bfloat16, device="cuda")
    K.moe_grouped(h, w1, w2, idx, y, in_w=in_w if act == "clamped" else None, limit=2.0 ** 120, alpha=1.0)
    exact = _exact(h, w1, w2, idx, act, in_w, 2.0 ** 120, 1.0, 0.0)
    assert float(exact.abs().min()) > 1e-8
    # two roundings to bfloat16 (the second of a value that has been rounded); the 32-bit evaluation is exact to 2^-20
    assert bool(((y.double() - exact).abs() <= 2.0 ** -8 * exact.abs()).all())


@pytest.mark.parametrize("params", [dict(activation="swiglu"), dict(activation="relu2"), dict(activation="clamped", limit=1.5, alpha=1.702, up_offset=1.0),
                                    dict(activation="swiglu", weight_input=True)])
def test_few_tokens_of_a_layer_grouped_and_one_by_one(monkeypatch, params):
    """Below 32 tokens a layer multiplies its experts grouped where that spares enough bytes: with the threshold at zero and out of
    reach, the same outputs up to their roundings."""
    from dryft_b200.ops import kernels as K
    from dryft_b200.parts.base import FFNS, Runtime, StepContext
    from dryft_b200.parts.moe import MoE
    from dryft_b200.weights import RandomSource

    params = dict(params, hidden_size=128, intermediate_size=64, experts=8, top=3)
    cls = FFNS.get("moe")
    dev = torch.device("cuda:0")

    def layer(threshold):
        monkeypatch.setattr(MoE, "GROUPED_SPARES_BYTES", threshold)
        rt = Runtime(dtype=torch.bfloat16, device=dev)
        return cls(params, "f.", RandomSource(cls.tensors(params, "f."), 5, torch.bfloat16, dev, std=0.1), rt)

    grouped, single = layer(0.0), layer(1e18)
    calls = []
    real = K.moe_grouped
    monkeypatch.setattr(K, "moe_grouped", lambda *a, **k: (calls.append(a[0].shape[0]), real(*a, **k)))
    for n in (1, 2, 5, 16, 17, 31, 32):
        h = torch.randn(n, 128, device="cuda").bfloat16()
        ints = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        ctx = StepContext(n_tokens=n, n_seqs=1, tokens=ints[:n], cu_q=ints[:2], seq_slot=ints[:1], tok_slot=ints[:n], tok_pos=ints[:n], decode=False)
        with torch.inference_mode():
            del calls[:]
            a = grouped.forward(h, ctx)
            assert calls == [n]
            b = single.forward(h, ctx)
            assert calls == [n] + [n] * (n >= 32)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                c = grouped.forward(h, ctx)
            graph.replay()
        assert torch.isfinite(a).all() and torch.equal(a, c)
        # activation, expert's row and weighted sum are rounded to bfloat16 on either side, each half a unit in 2^8
        assert float((a.double() - b.double()).norm() / b.double().norm()) < 6.0 * 2.0 ** -9, n
    K.check_error_flags()


def test_few_tokens_grouped_in_decode_steps(monkeypatch):
    """The same inside a model's decode steps: captured and eager give the same bits, and stay within bfloat16 of the other form."""
    import copy

    from dryft_b200.config import preset
    from dryft_b200.engine.api import Engine
    from dryft_b200.ops import kernels as K
    from dryft_b200.parts.moe import MoE

    cfg = copy.deepcopy(preset("tevovik-tiny"))
    for one in cfg["layers"]:
        one["mlp"]["expert"]["ff"] = 64
    logits = {}
    for threshold in (0.0, 1e18):
        monkeypatch.setattr(MoE, "GROUPED_SPARES_BYTES", threshold)
        for graphs in (True, False):
            eng = Engine.from_config(cfg, seed=3, dtype="bfloat16", max_batch=8, max_seq_len=256, max_tokens=1024, cuda_graphs=graphs)
            with torch.inference_mode():
                slots = eng.cache.open_sequences(5)
                eng.stepper.step(slots, [[1, 2, 3], [4] * 9, [5], [6, 7], [8] * 40], [[]] * 5)
                out = []
                for t in range(8):
                    at = torch.tensor(slots, device="cuda")
                    eng.cache.last_token.index_copy_(0, at, torch.tensor([t + 1, 2 * t, 3, 9, t], dtype=torch.int32, device="cuda"))
                    out.append(eng.stepper.decode_from_state(slots)[:5].clone())
            logits[threshold, graphs] = torch.stack(out)
    assert torch.isfinite(logits[0.0, True]).all()
    assert torch.equal(logits[0.0, True], logits[0.0, False]) and torch.equal(logits[1e18, True], logits[1e18, False])
    a, b = logits[0.0, True].double(), logits[1e18, True].double()
    # roundings of three layers of experts, some of which decide a router's close call the other way: most logits agree closely
    err = (a - b).norm(dim=-1) / b.norm(dim=-1)
    assert float(err.median()) < 3e-2, err
    K.check_error_flags()


@pytest.mark.parametrize("e,rows,width,f,launches", [(32, 1025, 128, 64, 3), (32, 1024, 128, 64, 4), (33, 1025, 128, 64, 4), (32, 1025, 192, 64, 4),
                                                     (8, 2048, 64, 128, 3)])
def test_many_rows_of_a_few_small_experts_run_on_mma_sync(e, rows, width, f, launches):
    from dryft_b200.ops import kernels as K

    h, w1, w2, idx, in_w = _case(rows, 1, e, width, f, "silu")
    y, plain = (torch.empty(rows, width, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    before = K.launch_count
    K.moe_grouped(h, w1, w2, idx, y)
    assert K.launch_count - before == launches
    K.moe_grouped(h, w1, w2, idx, plain, tcgen05=False)
    _check(y, _exact(h, w1, w2, idx, "silu", in_w, 0, 0, 0))
    assert launches != 3 or torch.equal(y, plain)
