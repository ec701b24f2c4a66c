"""What users of this library have it do, as cases that can be timed: requests to an ``Engine`` and feed-forwards of experts.

A *request* is a batch of prompts taken through the step function and gone on with for ``new`` tokens through the decode steps,
from free slots to slots given back.  In bfloat16 the tokens that follow are given (a recorded conversation is gone through
again), so that a token chosen the other way in a close call does not turn the rest into another conversation; in 32-bit the
tokens are the engine's own choice.  Every step's logits are the result.  A request with ``new == 0`` is a prompt step alone.

The *feed-forward* cases run one mixture of experts through the parts' own interface, which is what a model put together from
the registries does in every layer.  They are measured alone because a whole bfloat16 model of experts amplifies rounding: a
router's close call decided the other way is a different expert, hence a different and equally right logit.

The 4B and 8B shapes run with some of their layers (``layers``): every layer is like the next, and over all of them bfloat16
rounding alone moves a random model's logits by 3 to 5 parts in a hundred, too much to compare two correct implementations by.

Weights are random (there is no checkpoint here), the same for every seed; prompts, continuations and activations are the seed's."""

import math
import random

import torch

from dryft_b200 import Engine
from dryft_b200.config import config_from_dict, preset
from dryft_b200.parts.base import FFNS, Runtime, StepContext
from dryft_b200.sampling.sampler import SamplingParams, choose
from dryft_b200.weights import RandomSource, expected_tensors

WEIGHT_SEED = 11
DEVICE = "cuda:0"

# What an engine of each shape is built for: sequences at a time, the longest of them, tokens in the cache.
CAPACITY = {
    "qwen3-1k": (64, 4096, 32768),
    "qwen3-2k": (64, 4096, 32768),
    "qwen3-4b": (64, 8192, 32768),
    "qwen3-8b": (16, 8192, 32768),
    "vobusun-2k": (16, 4096, 16384),
    "dusupel-2k": (16, 4096, 16384),
}


def listed():
    request = {"kind": "request", "dtype": "bfloat16", "layers": 0, "ragged": False}
    return [
        # a short question to a small model: every launch is short, so their number and the gaps between them count
        dict(request, name="small-b1", model="qwen3-1k", batch=1, prompt=20, new=24),
        # one user of the 4B shape: a page of text and an answer, token by token
        dict(request, name="4b-b1", model="qwen3-4b", layers=8, batch=1, prompt=512, new=32),
        # the benchmark's batch of eight users
        dict(request, name="4b-b8", model="qwen3-4b", layers=8, batch=8, prompt=150, new=32, ragged=True),
        # a busy server: many users, short turns of unequal lengths
        dict(request, name="4b-b48", model="qwen3-4b", layers=8, batch=48, prompt=90, new=32, ragged=True),
        # the benchmark's prompt: how long until the first token
        dict(request, name="4b-prompt", model="qwen3-4b", layers=8, batch=1, prompt=2048, new=0),
        # prompts of unequal, odd lengths arriving together
        dict(request, name="4b-prompts", model="qwen3-4b", layers=8, batch=13, prompt=777, new=0, ragged=True),
        # two long documents and short summaries of them by the 8B shape
        dict(request, name="8b-long", model="qwen3-8b", layers=6, batch=2, prompt=3500, new=24),
        # the 32-bit path, as one checks a checkpoint with
        dict(request, name="small-f32", model="qwen3-1k", batch=4, prompt=200, new=8, ragged=True, dtype="float32"),
        # two of the other designs: linear attention, latents and a gated recurrence; delta rules and windows
        dict(request, name="vobusun-b1", model="vobusun-2k", batch=1, prompt=1300, new=16),
        dict(request, name="dusupel-b4", model="dusupel-2k", batch=4, prompt=400, new=12, ragged=True),
        # a layer of experts: a prompt's tokens, and a decode step's
        {"name": "experts-prompt", "kind": "experts", "model": "tevovik-2k", "tokens": 2048},
        {"name": "experts-decode", "kind": "experts", "model": "kerirax-2k", "tokens": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.25:
        return {"kind": "experts", "model": rng.choice(["tevovik-2k", "kerirax-2k", "tevovik-1k", "kerirax-1k"]), "tokens": _log_int(rng, 1, 4096)}
    case = {"kind": "request", "dtype": "bfloat16", "layers": 0, "ragged": rng.random() < 0.6}
    if pick < 0.35:
        batch = _log_int(rng, 1, 8)
        return dict(case, model="qwen3-1k", dtype="float32", batch=batch, prompt=_log_int(rng, 5, 800 // batch), new=rng.randint(1, 10))
    if pick < 0.5:
        batch = _log_int(rng, 1, 8)
        return dict(case, model=rng.choice(["vobusun-2k", "dusupel-2k"]), batch=batch, prompt=_log_int(rng, 20, 1600 // batch), new=rng.randint(0, 16))
    model = rng.choice(["qwen3-1k", "qwen3-2k", "qwen3-4b", "qwen3-4b"])
    case["layers"] = 8 if model == "qwen3-4b" else 0
    if rng.random() < 0.35:      # prompts alone
        batch = _log_int(rng, 1, 16)
        return dict(case, model=model, batch=batch, prompt=_log_int(rng, max(30, 200 // batch), 4000 // batch), new=0)
    batch = _log_int(rng, 1, 64)
    return dict(case, model=model, batch=batch, prompt=_log_int(rng, 16, max(32, 2500 // batch)), new=rng.randint(4, 20))


# ----------------------------------------------------------------------------- what a case's inputs are
def _lengths(case):
    """The prompts' lengths: all alike, or spread between an eighth of ``prompt`` and all of it (the same for every seed)."""
    b, p = case["batch"], case["prompt"]
    if not case["ragged"] or b == 1:
        return [p] * b
    lo = max(1, p // 8)
    return [p - int((p - lo) * ((i * 0.6180339887) % 1.0)) for i in range(b)]


def _tokens(case, seed):
    """(prompts, continuation ``new x batch``): seeded uniform token ids."""
    rng = random.Random(seed * 7919 + 17)
    vocab = _config(case["model"]).model_spec().vocab_size
    prompts = [[rng.randrange(vocab) for _ in range(n)] for n in _lengths(case)]
    return prompts, [[rng.randrange(vocab) for _ in range(case["batch"])] for _ in range(case["new"])]


def _shape(model, layers=0):
    """The shape's ``config.json``; ``layers``: that many of its layers (0: all)."""
    return dict(preset(model), num_hidden_layers=layers) if layers else preset(model)


def _config(model, layers=0):
    return config_from_dict(_shape(model, layers))


def _hidden(case, seed):
    """A step's normed activations, ``[tokens, width]``."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 104729 + 5)
    width = _config(case["model"]).model_spec().hidden_size
    return torch.randn(case["tokens"], width, generator=gen, device=DEVICE).to(torch.bfloat16)


def _experts_layer(model):
    """The first layer of the shape that is routed: (parameters, tensor prefix)."""
    for layer in _config(model).model_spec().layers:
        if layer.ffn is not None and layer.ffn.kind == "moe":
            return layer.ffn.params, layer.ffn_prefix
    raise ValueError(model)


def _experts_source(model):
    params, prefix = _experts_layer(model)
    return RandomSource(FFNS.get("moe").tensors(params, prefix), WEIGHT_SEED, torch.bfloat16, torch.device(DEVICE))


# ----------------------------------------------------------------------------- the state a program keeps
_kept = {}      # engines and layers by what they were built from: a program builds each once and sends it all its requests


def _engine(model, layers, dtype):
    key = ("engine", model, layers, dtype)
    if key not in _kept:
        batch, longest, tokens = CAPACITY[model]
        _kept[key] = Engine.from_config(_shape(model, layers), seed=WEIGHT_SEED, dtype=dtype, max_batch=batch, max_seq_len=longest, max_tokens=tokens)
    return _kept[key]


def _experts(model):
    key = ("experts", model)
    if key not in _kept:
        params, prefix = _experts_layer(model)
        rt = Runtime(dtype=torch.bfloat16, device=torch.device(DEVICE), sm_count=torch.cuda.get_device_properties(0).multi_processor_count)
        _kept[key] = FFNS.get("moe")(params, prefix, _experts_source(model), rt)
    return _kept[key]


def prepare(case, seed):
    if case["kind"] == "experts":
        n = case["tokens"]
        ints = torch.zeros(n + 1, dtype=torch.int32, device=DEVICE)
        ctx = StepContext(n_tokens=n, n_seqs=1, tokens=ints[:n], cu_q=ints[:2], seq_slot=ints[:1], tok_slot=ints[:n], tok_pos=ints[:n], decode=False)
        return {"case": case, "layer": _experts(case["model"]), "h": _hidden(case, seed), "ctx": ctx}
    prompts, after = _tokens(case, seed)
    eng = _engine(case["model"], case["layers"], case["dtype"])
    follow = torch.tensor(after, dtype=torch.int32).reshape(case["new"], case["batch"]).to(DEVICE)
    return {"case": case, "engine": eng, "prompts": prompts, "want": [[len(p) - 1] for p in prompts], "follow": follow}


def run(state):
    if state["case"]["kind"] == "experts":
        with torch.inference_mode():
            return state["layer"].forward(state["h"], state["ctx"])
    eng, new, batch = state["engine"], state["case"]["new"], state["case"]["batch"]
    given = state["case"]["dtype"] == "bfloat16"
    with torch.inference_mode():
        slots = eng.cache.open_sequences(batch)
        try:
            logits = eng.stepper.step(slots, state["prompts"], state["want"])
            if new == 0:
                return logits
            every = torch.empty((new + 1, batch, logits.shape[1]), dtype=torch.float32, device=DEVICE)
            chosen = torch.empty((new, batch), dtype=torch.int32, device=DEVICE)
            at = torch.tensor(slots, dtype=torch.int32).to(DEVICE)
            place = at.long()
            every[0].copy_(logits[:batch])
            for t in range(new):
                if given:
                    eng.cache.last_token.index_copy_(0, place, state["follow"][t])
                else:
                    choose(logits[:batch], SamplingParams(), row_slot=at, last_token=eng.cache.last_token, out=chosen[t])
                logits = eng.stepper.decode_from_state(slots)
                every[t + 1].copy_(logits[:batch])
        finally:
            eng.cache.close_sequences(slots)
    return every if given else {"logits": every, "tokens": chosen}


# ----------------------------------------------------------------------------- bytes, flops, tolerances
def work(case):
    if case["kind"] == "experts":
        params, _ = _experts_layer(case["model"])
        n, width, ff, experts, top = case["tokens"], params["hidden_size"], params["intermediate_size"], params["experts"], params["top"]
        read = experts * (1.0 - (1.0 - top / experts) ** n)      # experts that n tokens choose, on the mean
        return {"bytes": 2 * (read * 3 * width * ff + experts * width + 2 * n * width), "flops": 2 * n * (top * 3 * width * ff + experts * width)}
    cfg = _config(case["model"], case["layers"])
    spec = cfg.model_spec()
    size = 4 if case["dtype"] == "float32" else 2
    lens, new, b = _lengths(case), case["new"], case["batch"]
    weights = sum(math.prod(t.shape) for t in expected_tensors(spec).values() if t.kind == "matrix")      # each tensor once a step
    if not any("lm_head" in n or n == "head" for n in expected_tensors(spec)):
        weights += spec.vocab_size * spec.hidden_size
    kv = pairs = 0
    for step, layer in ((st, spec.layers[st.layer]) for st in spec.schedule):
        p = layer.mixer.params
        heads, dim = p.get("num_heads", 0), p.get("head_dim", p.get("qk_dim", 0)) or 0
        if layer.mixer.kind == "attention":
            kv += 2 * p["num_kv_heads"] * dim * size
            pairs += 4 * heads * dim
    seen = sum(n + t for n in lens for t in range(1, new + 1))      # cached tokens that the decode steps read
    flops = cfg.matmul_flops_per_token() * (sum(lens) + new * b) + 2 * spec.vocab_size * spec.hidden_size * b * (new + 1)
    flops += pairs * (sum(n * (n + 1) // 2 for n in lens) + seen)
    moved = (new + 1) * weights * size + kv * (sum(lens) + seen + new * b) + 4 * (new + 1) * b * spec.vocab_size
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """About four times what the path is off 64 bits, or what its sums in another order change; never more than 3 in a hundred
    (a step of the 4B shape's 8 layers is about 2 off, in whichever order it sums)."""
    if case["kind"] == "experts":
        return {"rel": 1e-2}
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "differ": 0.01}
    return {"rel": 0.02 if case["model"].startswith("vobusun") else 0.03}


# ----------------------------------------------------------------------------- the same in 64 bits
F = torch.float64


class _Weights:
    """A shape's weights by name, in 64 bits, each widened when it is asked for."""

    def __init__(self, model, layers, engine_dtype):
        self.expected = expected_tensors(_config(model, layers).model_spec())
        self.source = RandomSource(self.expected, WEIGHT_SEED, engine_dtype, torch.device(DEVICE))

    def __getitem__(self, name):
        return self.source.load(name, self.expected[name].kind).to(F)


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, dims, base, interleaved=False):
    """Rotary positions 0.. on the first ``dims`` of the last axis of ``[tokens, heads, dim]``."""
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=F, device=x.device) / dims)
    ang = torch.arange(x.shape[0], dtype=F, device=x.device)[:, None, None] * f
    c, s = torch.cos(ang), torch.sin(ang)
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if interleaved else (x[..., :half], x[..., half:dims])
    u, v = a * c - b * s, b * c + a * s
    y = torch.stack((u, v), -1).flatten(-2) if interleaved else torch.cat((u, v), -1)
    return torch.cat((y, x[..., dims:]), -1)


def _attend(q, k, v, scale, seen):
    """``q [n, heads, d]``, ``k [n, kv heads, d]``, ``v [n, kv heads, dv]`` -> ``[n, heads * dv]``; ``seen [n, n]``."""
    group = q.shape[1] // k.shape[1]
    out = []
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // group].T) * scale
        out.append(torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, h // group])
    return torch.cat(out, -1)


def _visible(n, window=None, keep=0):
    i, j = torch.arange(n, device=DEVICE)[:, None], torch.arange(n, device=DEVICE)[None, :]
    return (j <= i) if window is None else (j <= i) & ((i - j < window) | (j < keep))


def _qwen3(case, w, prompts):
    """Final normed rows of every sequence (layer by layer, so that each weight is widened once)."""
    cfg = _shape(case["model"], case["layers"])
    dim, eps, theta = cfg["head_dim"], cfg["rms_norm_eps"], cfg["rope_theta"]
    cut = [len(p) for p in prompts]
    x = w["model.embed_tokens.weight"][torch.tensor(sum(prompts, []), device=DEVICE)]
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        h = _unit(x, eps) * w[p + "input_layernorm.weight"]
        q, k, v = ((h @ w[p + "self_attn.%s_proj.weight" % c].T).view(len(h), -1, dim) for c in "qkv")
        q, k = _unit(q, eps) * w[p + "self_attn.q_norm.weight"], _unit(k, eps) * w[p + "self_attn.k_norm.weight"]
        o = [_attend(_turn(a, dim, theta), _turn(b, dim, theta), c, dim ** -0.5, _visible(len(a)))
             for a, b, c in zip(q.split(cut), k.split(cut), v.split(cut))]
        x = x + torch.cat(o) @ w[p + "self_attn.o_proj.weight"].T
        h = _unit(x, eps) * w[p + "post_attention_layernorm.weight"]
        x = x + (_silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    x = _unit(x, eps) * w["model.norm.weight"]
    return x.split(cut), w["model.embed_tokens.weight"] if cfg["tie_word_embeddings"] else w["lm_head.weight"]


def _conv(u, weight, bias=None):
    """A causal convolution per channel; the last tap meets the current token."""
    taps = weight.shape[1]
    padded = torch.cat((u.new_zeros(taps - 1, u.shape[1]), u))
    out = sum(padded[j:j + len(u)] * weight[:, j] for j in range(taps))
    return out if bias is None else out + bias


def _vobusun(case, w, prompts):
    cfg = preset(case["model"])
    eps, mult, streams = cfg["norm"]["eps"], cfg["residual_mult"], cfg["streams"]

    def owner(i):
        while cfg["layers"][i].get("weights_of") is not None:
            i = cfg["layers"][i]["weights_of"]
        return i

    def retention(m, p, h):
        n, heads, d, dv = len(h), m["heads"], m["dim"], m["vdim"]
        q, k, v = (h @ w[p + "q"].T).view(n, heads, d), (h @ w[p + "k"].T).view(n, heads, d), (h @ w[p + "v"].T).view(n, heads, dv)
        q, k = _turn(q, m["rot"]["dims"], m["rot"]["base"]), _turn(k, m["rot"]["dims"], m["rot"]["base"]) * d ** -0.5
        back = (torch.arange(n, device=DEVICE)[:, None] - torch.arange(n, device=DEVICE)[None, :])
        o = torch.stack([((q[:, a] @ k[:, a].T) * torch.where(back >= 0, m["decay"][a] ** back.clamp(min=0).to(F), 0.0)) @ v[:, a] for a in range(heads)], 1)
        return (_unit(o, eps).reshape(n, -1) * _silu(h @ w[p + "g"].T)) @ w[p + "o"].T

    def latent(m, p, h):
        n, heads, d, dr, r = len(h), m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        q = ((_unit(h @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T).view(n, heads, d + dr)
        low = h @ w[p + "dkv"].T
        c = _unit(low[:, :r], eps) * w[p + "dkv.norm"]
        turned = _turn(low[:, None, r:], m["rot"]["dims"], m["rot"]["base"], True).expand(n, heads, dr)
        q = torch.cat((q[..., :d], _turn(q[..., d:], m["rot"]["dims"], m["rot"]["base"], True)), -1)
        k = torch.cat(((c @ w[p + "uk"].T).view(n, heads, d), turned), -1)
        o = _attend(q, k, (c @ w[p + "uv"].T).view(n, heads, m["vdim"]), m["scale"], _visible(n, m["mask"]["size"]))
        return (o.view(n, heads, -1) * torch.sigmoid(h @ w[p + "g"].T)[..., None]).reshape(n, -1) @ w[p + "o"].T

    def gated_recurrence(m, p, h):
        n, width, blocks = len(h), m["width"], m["blocks"]
        z = h @ w[p + "y"].T + w[p + "y.b"]
        y = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
        u = _conv(h @ w[p + "x"].T + w[p + "x.b"], w[p + "conv"], w[p + "conv.b"])
        ub = u.view(n, blocks, width // blocks)
        r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, w[p + c].view(blocks, width // blocks, width // blocks)) + w[p + c + ".b"].view(blocks, -1)).reshape(n, width) for c in ("ra", "ri"))
        a = torch.exp(-8.0 * r * torch.nn.functional.softplus(w[p + "lam"]))
        s, out, add = torch.zeros(width, dtype=F, device=DEVICE), [], torch.sqrt(1.0 - a * a) * i * u
        for t in range(n):
            s = a[t] * s + add[t]
            out.append(s)
        return (torch.stack(out) * y) @ w[p + "o"].T

    mixers = {"retention": retention, "latent_attention": latent, "rglru": gated_recurrence}
    rows = []
    for ids in prompts:
        t = torch.tensor(ids, device=DEVICE)
        pair = cfg["embedding"]["bigram"]
        hashed = torch.cat((t.new_full((1,), pair["buckets"]), (t[:-1] * pair["mul_prev"] + t[1:] * pair["mul_cur"]) % pair["buckets"]))
        xs = (_unit(w["embed"][t] * cfg["embedding"]["scale"] + w["bigram"][hashed], eps) * w["embed.norm"]).expand(streams, -1, -1)
        for i, layer in enumerate(cfg["layers"]):
            p = "l%d." % owner(i)
            for q in (1, 2):
                h = _unit(torch.einsum("s,snw->nw", w[p + "hc%d.in" % q], xs), eps) * w[p + "norm%d" % q]
                if q == 1:
                    y = mixers[layer["type"]](layer["mixer"], p + "mix.", h)
                else:
                    limit = layer["mlp"]["limit"]
                    g, u = (h @ w[p + "mlp.gate"].T).clamp(max=limit), (h @ w[p + "mlp.up"].T).clamp(min=-limit, max=limit)
                    y = (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[p + "mlp.down"].T
                xs = torch.einsum("st,snw->tnw", w[p + "hc%d.mix" % q], xs) + mult * w[p + "hc%d.out" % q][:, None, None] * y
        rows.append(_unit(xs.sum(0), eps) * w["final.norm"])
    return rows, w["head"]


def _dusupel(case, w, prompts):
    cfg = preset(case["model"])
    eps, mult, loop = cfg["norm"]["eps"], cfg["residual_mult"], cfg["loop"]
    order = list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], len(cfg["layers"])))

    def layer_norm(x, name):
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w[name], w[name + ".b"], eps)

    def attention(m, p, h):
        n = len(h)
        q, k, v = (_conv(h @ w[p + c].T, w[p + c + ".conv"]).view(n, -1, m["vdim"] if c == "v" else m["dim"]) for c in "qkv")
        q, k = _turn(q, m["rot"]["dims"], m["rot"]["base"]), _turn(k, m["rot"]["dims"], m["rot"]["base"])
        o = _attend(q, k, v, m["scale"], _visible(n, m["mask"]["size"], m["mask"]["keep_first"]))
        return (o * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T

    def delta(m, p, h, per_channel):
        n, heads, groups, d, dv = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(_conv(h @ w[p + c].T, w[p + c + ".conv"])) for c in "qkv")
        q, k = (x.view(n, groups, d) / torch.sqrt((x.view(n, groups, d) ** 2).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        q, k, v = (q * d ** -0.5).repeat_interleave(heads // groups, 1), k.repeat_interleave(heads // groups, 1), v.view(n, heads, dv)
        beta = torch.sigmoid(h @ w[p + "b"].T)
        if per_channel:
            z = torch.nn.functional.softplus((h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "dt_bias"].reshape(-1)).view(n, heads, d)
            keep, gate = torch.exp(-torch.exp(w[p + "A_log"]).view(heads, 1) * z), torch.sigmoid((h @ w[p + "g1"].T) @ w[p + "g2"].T)
        else:
            z = torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"])
            keep, gate = torch.exp(-torch.exp(w[p + "A_log"]) * z)[..., None], _silu(h @ w[p + "g"].T)
        s, out = torch.zeros(heads, d, dv, dtype=F, device=DEVICE), []
        for t in range(n):
            s = keep[t][:, :, None] * s
            u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", s, k[t]))
            s = s + k[t][:, :, None] * u[:, None, :]
            out.append(torch.einsum("hdv,hd->hv", s, q[t]))
        return ((_unit(torch.stack(out), eps) * w[p + "norm"]).reshape(n, -1) * gate) @ w[p + "o"].T

    rows = []
    for ids in prompts:
        x = w["embed"][torch.tensor(ids, device=DEVICE)]
        for i in order:
            layer, p = cfg["layers"][i], "l%d." % i
            h = layer_norm(x, p + "norm1")
            if layer["type"] == "parallel":
                m = layer["mixer"]
                y = m["left_scale"] * attention(m["left"], p + "mix.left.", h) + m["right_scale"] * delta(m["right"], p + "mix.right.", h, False)
            else:
                y = delta(layer["mixer"], p + "mix.", h, True)
            h = layer_norm(x, p + "norm2")
            x = x + mult * (y + (_silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T)
        rows.append(layer_norm(x, "final.norm"))
    return rows, w["head"]


def _exact_experts(case, seed):
    params, prefix = _experts_layer(case["model"])
    names = params.get("names") or {}
    src, h = _experts_source(case["model"]), _hidden(case, seed).to(F)
    expert = prefix + names.get("expert", "experts.{}.")
    gate, up, down = names.get("gate", "gate_proj.weight"), names.get("up", "up_proj.weight"), names.get("down", "down_proj.weight")
    z = h @ src.load(prefix + names.get("router", "router.weight"), "matrix").to(F).T
    if params.get("router_bias"):
        z = z + src.load(prefix + names.get("router_bias", "router.bias"), "vector").to(F)
    score = torch.sigmoid(z) if params.get("score", "softmax") == "sigmoid" else torch.softmax(z, -1)
    n, e = score.shape
    groups, keep = params.get("groups", 1), params.get("keep", params.get("groups", 1))
    best = score.view(n, groups, -1).amax(-1).topk(keep, -1).indices
    allowed = torch.zeros(n, groups, dtype=torch.bool, device=DEVICE).scatter_(1, best, True).repeat_interleave(e // groups, 1)
    chosen = score.masked_fill(~allowed, -1.0).topk(params["top"], -1).indices
    weight = score.gather(1, chosen)
    if params.get("renormalize"):
        weight = weight / (weight.sum(-1, keepdim=True) + params.get("renorm_eps", 0.0))
    out = torch.zeros_like(h)
    clamped = params.get("activation", "swiglu") == "clamped"
    limit, alpha, offset = params.get("limit"), params.get("alpha", 1.0), params.get("up_offset", 0.0)
    for i in range(e):
        t, k = torch.nonzero(chosen == i, as_tuple=True)
        if not len(t):
            continue
        p = expert.format(i)
        x, by = h[t], weight[t, k][:, None]
        if params.get("weight_input"):
            x, by = x * by, 1.0
        g, u = x @ src.load(p + gate, "matrix").to(F).T, x @ src.load(p + up, "matrix").to(F).T
        if clamped:
            if limit is not None:
                g, u = g.clamp(max=limit), u.clamp(min=-limit, max=limit)
            a = g * torch.sigmoid(alpha * g) * (u + offset)
        else:
            a = _silu(g) * u
        out.index_add_(0, t, (a @ src.load(p + down, "matrix").to(F).T) * by)
    return out


def exact(case, seed):
    with torch.inference_mode():
        if case["kind"] == "experts":
            return _exact_experts(case, seed)
        prompts, after = _tokens(case, seed)
        dtype = getattr(torch, case["dtype"])
        w = _Weights(case["model"], case["layers"], dtype)
        forward = {"qwen3": _qwen3, "vobusun": _vobusun, "dusupel": _dusupel}[case["model"].split("-")[0]]
        new, chosen = case["new"], []
        if dtype == torch.float32:      # the engine's own choices: one whole evaluation for each
            for _ in range(new):
                rows, head = forward(case, w, [p + [c[b] for c in chosen] for b, p in enumerate(prompts)])
                chosen.append([int(torch.argmax(head @ r[-1])) for r in rows])
            after = chosen
        rows, head = forward(case, w, [p + [a[b] for a in after] for b, p in enumerate(prompts)])
        every = torch.stack([r[len(r) - 1 - new:] for r in rows], 1) @ head.T      # [new + 1, batch, vocab]
        if new == 0:
            return every[0]
        return every if dtype == torch.bfloat16 else {"logits": every, "tokens": None}
