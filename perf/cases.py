"""The work that this framework is measured by: prompts read and tokens decoded through the step function.

A pass serves a set of requests from their admission to their end through ``ModelRunner.step``, as the engine's
loop and ``bin/trace_run`` drive it: prompts in portions of at most ``step_tokens`` tokens a step, then ``new``
decode steps (the tokens are given, so that two implementations compute the same thing), then every request is
finished.  What comes back are the logits behind each request's last token.

A case's fields: ``model`` (a published LFM2 shape, or one of the other designs at the width that ``bench.py``
runs it at), ``dtype``, ``requests``, ``prompt`` (tokens of a prompt; ``ragged``: of the longest, the others go
down to a quarter of it), ``step_tokens``, ``new``, and ``streamed``: whether the requests arrive together, or
one after the other while those before them decode (continuous batching).
"""
from __future__ import annotations

import math

import torch

from neurogrid_b200.config import config_from_dict
from neurogrid_b200.engine import ModelRunner, StepEntry
from neurogrid_b200.engine.loading import parse_dtype, require_cuda
from neurogrid_b200.models import build_model, declare_tensors

DEVICE = "cuda:0"
VOCAB = 65536
PAGE = 16

_LFM2_LAYERS = ["conv", "conv", "full_attention", "conv", "conv", "full_attention", "conv", "conv", "full_attention",
                "conv", "full_attention", "conv", "full_attention", "conv", "full_attention", "conv"]
_LFM2_SHAPES = {"lfm2-350m": (1024, 16, 6656), "lfm2-700m": (1536, 24, 10240), "lfm2-1.2b": (2048, 32, 12288)}


# ------------------------------------------------------------------------------------------------ configurations
def _lfm2(name):
    hidden, heads, ff = _LFM2_SHAPES[name]
    return dict(architectures=["Lfm2ForCausalLM"], model_type="lfm2", vocab_size=VOCAB, hidden_size=hidden,
                num_hidden_layers=16, layer_types=list(_LFM2_LAYERS), num_attention_heads=heads, num_key_value_heads=8,
                block_ff_dim=ff, block_auto_adjust_ff_dim=True, block_multiple_of=256, block_ffn_dim_multiplier=1.0,
                conv_L_cache=3, conv_bias=False, tie_embedding=True, rope_theta=1000000.0, norm_eps=1e-5,
                max_position_embeddings=128000)


def _lfm2_ff(cfg):
    d, m = int(2 * cfg["block_ff_dim"] / 3), cfg["block_multiple_of"]
    return (d + m - 1) // m * m


def _metanex(width):
    heads = width // 128
    ret = {"type": "retention", "mixer": {"heads": heads, "dim": 128, "vdim": 128,
                                          "decay": [1.0 - 2.0 ** (-5 - 6 * h / max(1, heads - 1)) for h in range(heads)],
                                          "rot": {"dims": 64, "base": 1000000.0}}}
    lat = {"type": "latent_attention", "mixer": {"heads": heads, "dim": 128, "vdim": 128, "q_rank": 768, "kv_rank": 128,
                                                 "scale": 128 ** -0.5, "mask": {"size": 1024}}}
    mlp = {"kind": "moe", "router": {"experts": 16, "top": 4}, "expert": {"ff": width // 4}, "shared": {"ff": width // 2}}
    return {"architecture": "Metanex", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "canon": {"taps": 4},
            "token_side": {"dim": 64}, "layers": [dict((ret, ret, lat, ret)[i % 4], mlp=mlp) for i in range(16)]}


def _rofulorn(width):
    heads = width // 64
    ff = _lfm2_ff(_lfm2("lfm2-350m" if width == 1024 else "lfm2-1.2b"))
    a2 = {"type": "attention_2", "mixer": {"heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 64, "scale": 0.125,
                                           "mask": {"size": 1024}, "rot": {"dims": 32, "base": 1000000.0}}}
    diff = {"heads": heads // 2, "kv_heads": heads // 8, "dim": 64, "vdim": 128, "scale": 0.125, "softcap": 30.0,
            "diff": 0.5, "mask": {"size": 1024, "keep_first": 4},
            "rot": {"dims": 32, "base": 20000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 2048}}}
    layers = []
    for i in range(16):
        layer = dict(a2) if i % 2 == 0 else {"type": "attention", "mixer": dict(diff, **({"kv_from": i - 2} if i % 4 == 3 else {}))}
        layers.append(dict(layer, mlp={"kind": "dense", "ff": ff}))
    return {"architecture": "Rofulorn", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "embedding": {"scale": 0.5},
            "layers": layers}


def _config(model):
    family, size = model.split("-")
    return _lfm2(model) if family == "lfm2" else _metanex(int(size)) if family == "metanex" else _rofulorn(int(size))


# ------------------------------------------------------------------------------------------------ cases
def _case(model, requests, prompt, new, *, name=None, dtype="bfloat16", ragged=False, step_tokens=2048, streamed=False):
    c = dict(model=model, dtype=dtype, requests=requests, prompt=prompt, new=new, ragged=ragged,
             step_tokens=step_tokens, streamed=streamed)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short question to a small model: one request, a handful of tokens; latency and launches
        _case("lfm2-350m", 1, 19, 8, name="question"),
        # the headline: a batch of 8 behind prompts of 2,048 tokens
        _case("lfm2-1.2b", 8, 2048, 96, name="batch-8"),
        # a full server: many requests with short prompts of differing lengths
        _case("lfm2-1.2b", 64, 173, 32, name="batch-64", ragged=True),
        # time to the first token of one ordinary long prompt
        _case("lfm2-1.2b", 1, 2048, 0, name="prompt-2048"),
        # prompts of odd lengths that arrive together and are read in one step
        _case("lfm2-700m", 6, 611, 0, name="prompts-ragged", ragged=True, step_tokens=4096),
        # a document: 16,384 tokens in portions, then an answer begins
        _case("lfm2-700m", 1, 16384, 16, name="document"),
        # continuous batching: each step holds a portion of one prompt beside the decode tokens of the others
        _case("lfm2-1.2b", 12, 257, 8, name="stream", ragged=True, step_tokens=128, streamed=True),
        # the 32-bit path, which replays are checked with
        _case("lfm2-350m", 2, 96, 8, name="float32", dtype="float32"),
        # the designs beside LFM2 whose layers differ most from it: state and latent layers with routed experts ...
        _case("metanex-1024", 1, 2048, 0, name="metanex-prompt"),
        _case("metanex-2048", 8, 256, 48, name="metanex-batch-8"),
        # ... and windowed attention with 32-bit weights, one and two maps a head
        _case("rofulorn-2048", 1, 2048, 0, name="rofulorn-prompt"),
        _case("rofulorn-1024", 8, 512, 48, name="rofulorn-batch-8"),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges: each kind of work above with sizes of its own."""
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("turns", "turns", "prompt", "prompts", "document", "stream", "float32", "metanex", "rofulorn"))
        lfm2 = rng.choice(tuple(_LFM2_SHAPES))
        if kind == "turns":
            c = _case(lfm2, _log(rng, 1, 64), _log(rng, 16, 2048), _log(rng, 8, 96), ragged=rng.random() < 0.5)
        elif kind == "prompt":
            c = _case(lfm2, 1, _log(rng, 100, 4096), 0, step_tokens=4096)
        elif kind == "prompts":
            c = _case(lfm2, rng.randint(2, 8), _log(rng, 50, 512), 0, ragged=True, step_tokens=4096)
        elif kind == "document":
            c = _case(rng.choice(("lfm2-350m", "lfm2-700m")), 1, _log(rng, 4096, 16384), _log(rng, 4, 32))
        elif kind == "stream":
            c = _case(lfm2, rng.randint(3, 16), _log(rng, 64, 400), 8, ragged=True, step_tokens=rng.choice((64, 128, 256)), streamed=True)
        elif kind == "float32":
            c = _case("lfm2-350m", rng.randint(1, 4), _log(rng, 16, 160), rng.randint(4, 12), dtype="float32")
        else:
            model = "%s-%d" % (kind, rng.choice((1024, 2048)))
            c = (_case(model, 1, _log(rng, 256, 2048), 0) if rng.random() < 0.5 else
                 _case(model, _log(rng, 1, 8), _log(rng, 64, 1024), _log(rng, 8, 48)))
        shapes = [{k: v for k, v in x.items() if k != "name"} for x in listed()]
        if c not in shapes and _cost(c) <= most:
            return c


def _lengths(case):
    """Tokens of every prompt: the first is the longest, the others lie between a quarter of it and it."""
    n, p = case["requests"], case["prompt"]
    if not case["ragged"]:
        return [p] * n
    return [p if i == 0 else max(1, round(p * (0.25 + 0.75 * (i * 0.6180339887 % 1.0)))) for i in range(n)]


def _plan(case):
    """The steps of a pass: lists of (request, first token, tokens, wanted).  The steps that hold a request's last
    token are those whose logits come back."""
    lens, new, budget = _lengths(case), case["new"], case["step_tokens"]
    at = [0] * len(lens)
    steps = []
    if case["streamed"]:
        for i, n in enumerate(lens):
            while at[i] < n:
                step = [(j, at[j], 1, True) for j in range(i)]
                take = min(n - at[i], budget - len(step))
                step.append((i, at[i], take, at[i] + take == n))
                for j, _, k, _ in step:
                    at[j] += k
                steps.append(step)
    else:
        step, room = [], budget
        for i, n in enumerate(lens):
            while at[i] < n:
                take = min(n - at[i], room)
                step.append((i, at[i], take, at[i] + take == n))
                at[i] += take
                room -= take
                if room == 0:
                    steps.append(step)
                    step, room = [], budget
        if step:
            steps.append(step)
    for _ in range(new):
        steps.append([(j, at[j], 1, True) for j in range(len(lens))])
        at = [a + 1 for a in at]
    return steps, at


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


# ------------------------------------------------------------------------------------------------ inputs
def _std(name, shape):
    """Standard deviation of a drawn matrix of the other designs: products of order one, attention that is peaked and
    routers that decide, as training leaves them; matrices that write into the stream by 1 / sqrt(sublayers)."""
    leaf = name.split(".")[-1]
    gain = 2.0 if leaf in ("uq", "uk", "head") else 4.0 if leaf == "router" else 32 ** -0.5 if leaf in ("o", "down") else 1.0
    return gain / shape[-1] ** 0.5


def _weights(case, seed):
    """Name -> bfloat16 tensor, as a checkpoint holds them."""
    decls = declare_tensors(config_from_dict(_config(case["model"])).model_spec())
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    lfm2 = case["model"].startswith("lfm2")
    out = {}
    for name in sorted(decls):
        shape, init = decls[name].shape, decls[name].init
        t = torch.randn(shape, generator=gen, device=DEVICE)
        if lfm2:
            t = 1.0 + 0.1 * t if init == "norm" else t * (0.2 if init == "conv" else 0.02)
        elif len(shape) < 2:
            t = (0.2 if "side" in name else 1.0) * (1.0 + 0.1 * t) if "norm" in name else t * 0.1
        elif "canon" in name:
            t = 0.2 * t
        elif "embed" not in name:
            t = t * _std(name, shape)
        out[name] = t.to(torch.bfloat16)
    return out


def _tokens(case, seed):
    gen = torch.Generator().manual_seed(seed + 1)
    return [torch.randint(0, VOCAB, (n,), generator=gen).tolist() for n in _plan(case)[1]]


def prepare(case, seed):
    """A server that is up: the model's weights on the device, the runner with its cache, and two passes behind it,
    so that the graphs of the shapes it meets are there."""
    device, dtype = require_cuda(DEVICE), parse_dtype(case["dtype"])
    model = build_model(config_from_dict(_config(case["model"])).model_spec(), _weights(case, seed), dtype=dtype, device=device)
    steps, ends = _plan(case)
    tokens = _tokens(case, seed)
    longest = max(ends)
    runner = ModelRunner(model, num_pages=sum(-(-n // PAGE) for n in ends) + len(ends), page_size=PAGE,
                         max_requests=case["requests"], max_seq_len=-(-longest // PAGE) * PAGE,
                         max_tokens_per_step=max(case["step_tokens"], case["requests"]))
    last = {i: n for i, n in enumerate(ends)}
    asked = [([(i, tokens[i][a:a + n], [n - 1] if want else []) for i, a, n, want in step],
              any(a + n == last[i] for i, a, n, _ in step)) for step in steps]
    state = {"runner": runner, "steps": asked, "requests": range(len(ends))}
    for _ in range(2):
        run(state)
    runner.check_status()
    return state


def run(state):
    runner, kept = state["runner"], []
    final = len(state["steps"]) - 1
    for k, (entries, keep) in enumerate(state["steps"]):
        logits = runner.step([StepEntry(i, toks, want) for i, toks, want in entries])
        if keep:
            kept.append(logits if k == final else logits.clone())      # a step's logits live until the next step
    for i in state["requests"]:
        runner.finish(i)
    return kept


# ------------------------------------------------------------------------------------------------ what a pass needs
def _sizes(case):
    """(weight elements a step reads whatever its rows, elements per routed expert, experts, top, routed layers,
    attention layers as (key elements a token, score and value multiplies a query and key, window), state floats)."""
    c = _config(case["model"])
    if case["model"].startswith("lfm2"):
        H, ff = c["hidden_size"], _lfm2_ff(c)
        attn = sum(t == "full_attention" for t in c["layer_types"])
        body = 16 * 3 * H * ff + (16 - attn) * 4 * H * H + attn * (2 * H * H + 2 * 512 * H)
        return body, (0, 0, 0, 0), [(2 * 512, 2 * H, None)] * attn, (16 - attn) * 3 * H
    D = c["width"]
    body, attn, state, routed = 0, [], 0, (0, 0, 0, 0)
    for layer in c["layers"]:
        m = layer["mixer"]
        if layer["type"] == "retention":
            hd = m["heads"] * m["dim"]
            body += 5 * D * hd
            state += 2 * m["heads"] * m["dim"] * m["vdim"]
        elif layer["type"] == "latent_attention":
            hd = m["heads"] * m["dim"]
            body += D * (m["q_rank"] + m["kv_rank"] + m["heads"]) + hd * (m["q_rank"] + 2 * m["kv_rank"]) + hd * D
            attn.append((m["kv_rank"], 2 * m["heads"] * m["kv_rank"], 1024))
        else:
            maps = 2 if layer["type"] == "attention" else 1
            q, k, v = m["heads"] * maps * m["dim"], m["kv_heads"] * maps * m["dim"], m["kv_heads"] * m["vdim"]
            body += D * (q + m["heads"] * m["vdim"] + (0 if m.get("kv_from") is not None else k + v))
            attn.append((k + v, maps * m["heads"] * (m["dim"] + m["vdim"]), 1024))
        mlp = layer["mlp"]
        if mlp["kind"] == "moe":
            body += 3 * D * mlp["shared"]["ff"] + D * mlp["router"]["experts"] + 2 * D * 64
            routed = (3 * D * mlp["expert"]["ff"], mlp["router"]["experts"], mlp["router"]["top"], routed[3] + 1)
        else:
            body += 3 * D * mlp["ff"]
    return body, routed, attn, state


def work(case):
    """Each step reads every weight it needs once (they are larger than the L2), the keys, values and states of its
    requests, and writes its new keys and the wanted logits."""
    esz = 4 if case["dtype"] == "float32" else 2
    body, (per_expert, experts, top, routed), attn, state = _sizes(case)
    D = _config(case["model"]).get("hidden_size") or _config(case["model"])["width"]
    nbytes = flops = 0.0
    for step in _plan(case)[0]:
        rows, wanted = sum(n for _, _, n, _ in step), sum(w for *_, w in step)
        weights = body + (VOCAB * D if wanted else 0)
        if experts:
            weights += routed * per_expert * experts * (1.0 - (1.0 - top / experts) ** rows)
        nbytes += esz * weights + 4.0 * wanted * VOCAB + esz * rows * D + 4.0 * state * len(step)
        flops += 2.0 * rows * (body + routed * per_expert * top) + 2.0 * wanted * VOCAB * D
        for kv, mul, window in attn:
            for _, a, n, _ in step:
                seen = a + n if window is None else min(a + n, window + n)
                pairs = sum(min(t + 1, window) for t in range(a, a + n)) if window else n * a + n * (n + 1) / 2
                nbytes += esz * kv * (seen + n)
                flops += 2.0 * mul * pairs
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # 32 bits: 8e-6 from 64 bits.  bfloat16: two runs of one implementation, whose order of a few float32 sums is not
    # fixed, are 0.012 apart with LFM2 and 0.005 with the others (a last bit that falls the other way spreads through
    # sixteen layers; all matrices of LFM2 are drawn alike, which lets it grow)
    if case["dtype"] == "float32":
        return {"rel": 4e-5, "max": 1e-3}
    return {"rel": 0.03, "max": 0.5} if case["model"].startswith("lfm2") else {"rel": 0.02, "max": 0.3}


# ------------------------------------------------------------------------------------------------ in 64 bits
F64 = torch.float64


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _turn(x, freq, adjacent):
    """x [T, heads, dim]: the first 2 * len(freq) coordinates turn by position * freq, paired (2i, 2i + 1) or (i, i + half)."""
    n = freq.numel()
    a = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * freq
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    one, two = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if adjacent else (slice(0, n), slice(n, 2 * n))
    y = x.clone()
    y[..., one], y[..., two] = x[..., one] * c - x[..., two] * s, x[..., two] * c + x[..., one] * s
    return y


def _freq(dims, base, scaling=None):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEVICE) / dims)
    if scaling:
        wave, o = 2 * math.pi / f, scaling["original"]
        s = ((o / wave - scaling["low"]) / (scaling["high"] - scaling["low"])).clamp(0, 1)
        f = (1 - s) * f / scaling["factor"] + s * f
    return f


def _attend(q, k, v, scale, window=None, first=0, cap=None, block=2048):
    """Causal softmax attention, q [T, H, d], k [T, G, d], v [T, G, e]: head h reads key/value head h // (H / G)."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=q.device)
    j = torch.arange(T, device=q.device)
    for a in range(0, T, block):
        i = torch.arange(a, min(T, a + block), device=q.device)[:, None]
        hidden = j > i
        if window:
            hidden |= (i - j >= window) & (j >= first)
        for h in range(H):
            s = (q[a:a + block, h] @ k[:, h * G // H].T) * scale
            s = cap * torch.tanh(s / cap) if cap else s
            out[a:a + block, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ v[:, h * G // H]
    return out


def _taps(u, w):
    """Causal depthwise convolution of u [T, D] with w [D, L]."""
    L = w.shape[1]
    return sum(w[:, j] * torch.cat([u.new_zeros(L - 1 - j, u.shape[1]), u[:u.shape[0] - (L - 1 - j)]])[:u.shape[0]] for j in range(L))


def _lfm2_logits(c, w, tokens):
    H, heads, eps = c["hidden_size"], c["num_attention_heads"], c["norm_eps"]
    freq = _freq(64, c["rope_theta"])
    x = w["model.embed_tokens.weight"][tokens]
    T = x.shape[0]
    for i, kind in enumerate(c["layer_types"]):
        g = lambda name: w["model.layers.%d.%s.weight" % (i, name)]  # noqa: E731
        n = _rms(x, eps) * g("operator_norm")
        if kind == "conv":
            b, cc, u = (n @ g("conv.in_proj").T).split(H, -1)
            m = (cc * _taps(b * u, g("conv.conv").reshape(H, -1))) @ g("conv.out_proj").T
        else:
            q, k, v = ((n @ g("self_attn.%s_proj" % s).T).view(T, -1, 64) for s in "qkv")
            q = _turn(_rms(q, eps) * g("self_attn.q_layernorm"), freq, False)
            k = _turn(_rms(k, eps) * g("self_attn.k_layernorm"), freq, False)
            m = _attend(q, k, v, 0.125).reshape(T, heads * 64) @ g("self_attn.out_proj").T
        x = x + m
        n = _rms(x, eps) * g("ffn_norm")
        x = x + (_silu(n @ g("feed_forward.w1").T) * (n @ g("feed_forward.w3").T)) @ g("feed_forward.w2").T
    return (_rms(x[-1:], eps) * w["model.embedding_norm.weight"]) @ w["model.embed_tokens.weight"].T


def _retention(h, w, pre, m, eps):
    T, H, d, e = h.shape[0], m["heads"], m["dim"], m["vdim"]
    freq = _freq(m["rot"]["dims"], m["rot"]["base"])
    q = _turn((h @ w[pre + "q"].T).view(T, H, d), freq, False)
    k = _turn((h @ w[pre + "k"].T).view(T, H, d), freq, False) * d ** -0.5
    v = (h @ w[pre + "v"].T).view(T, H, e)
    t = torch.arange(T, dtype=F64, device=h.device)
    age = t[:, None] - t
    o = torch.stack([((q[:, i] @ k[:, i].T) * torch.where(age >= 0, m["decay"][i] ** age.clamp(min=0), 0.0)) @ v[:, i]
                     for i in range(H)], 1)
    return (_rms(o, eps).reshape(T, H * e) * _silu(h @ w[pre + "g"].T)) @ w[pre + "o"].T


def _latent(h, w, pre, m, eps):
    T, H, d, e = h.shape[0], m["heads"], m["dim"], m["vdim"]
    q = ((_rms(h @ w[pre + "dq"].T, eps) * w[pre + "dq.norm"]) @ w[pre + "uq"].T).view(T, H, d)
    c = _rms(h @ w[pre + "dkv"].T, eps) * w[pre + "dkv.norm"]
    o = _attend(q, (c @ w[pre + "uk"].T).view(T, H, d), (c @ w[pre + "uv"].T).view(T, H, e), m["scale"], m["mask"]["size"])
    return (o * torch.sigmoid(h @ w[pre + "g"].T)[:, :, None]).reshape(T, H * e) @ w[pre + "o"].T


def _experts(h, w, pre, mlp):
    def one(x, p):
        return (_silu(x @ w[p + "gate"].T) * (x @ w[p + "up"].T)) @ w[p + "down"].T
    val, idx = torch.topk(h @ w[pre + "router"].T + w[pre + "router.b"], mlp["router"]["top"], -1)
    p = torch.softmax(val, -1)
    out = one(h, pre + "shared.")
    for e in range(mlp["router"]["experts"]):
        rows, place = torch.nonzero(idx == e, as_tuple=True)
        out[rows] += p[rows, place][:, None] * one(h[rows], "%se%d." % (pre, e))
    return out


def _metanex_logits(c, w, tokens):
    eps, side = c["norm"]["eps"], c["token_side"]["dim"]
    x = w["embed"][tokens]
    for i, layer in enumerate(c["layers"]):
        p = "l%d." % i
        u = _rms(x, eps) * w[p + "norm1"]
        u = u + _taps(u, w[p + "canon1"])
        x = x + (_retention if layer["type"] == "retention" else _latent)(u, w, p + "mix.", layer["mixer"], eps)
        u = _rms(x, eps) * w[p + "norm2"]
        x = x + _experts(u + _taps(u, w[p + "canon2"]), w, p + "mlp.", layer["mlp"])
        y = (_gelu(x @ w[p + "side.gate"].T) * w["side.embed"][tokens, i * side:(i + 1) * side]) @ w[p + "side.proj"].T
        x = x + _rms(y, eps) * w[p + "side.norm"]
    return (_rms(x[-1:], eps) * w["final.norm"]) @ w["head"].T


def _mapped(h, w, pre, m, eps, two, held):
    """One map a head, or the difference of two over the same values; returns the keys and values it read as well."""
    T, H, G, d, e = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    freq, window, maps = _freq(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling")), m["mask"]["size"], 2 if two else 1

    def rows(s):
        return h @ w[pre + s].T + (w[pre + s + ".b"] if two else 0.0)

    def keys(s, n):
        z = rows(s).view(T, n * maps, d)
        return _turn(_rms(z, eps) * w[pre + s + ".norm"] if two else z, freq, True).view(T, n, maps, d)

    q = keys("q", H)
    k, v = held if held is not None else (keys("k", G), rows("v").view(T, G, e))
    a = [_attend(q[:, :, i], k[:, :, i], v, m["scale"], window, m["mask"].get("keep_first", 0), m.get("softcap")) for i in range(maps)]
    if two:
        lam = torch.exp((w[pre + "lq1"] * w[pre + "lk1"]).sum()) - torch.exp((w[pre + "lq2"] * w[pre + "lk2"]).sum()) + m["diff"]
        a = [_rms(a[0] - lam * a[1], eps) * (1.0 - m["diff"])]
    return a[0].reshape(T, H * e) @ w[pre + "o"].T + (w[pre + "o.b"] if two else 0.0), (k, v)


def _rofulorn_logits(c, w, tokens):
    eps, held = c["norm"]["eps"], {}

    def norm(x, g):
        x = x - x.mean(-1, keepdim=True)
        return _rms(x, eps) * g

    x = w["embed"][tokens] * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        h = norm(x, w[p + "norm1"])
        y, held[i] = _mapped(h, w, p + "mix.", m, eps, layer["type"] == "attention", held.get(m.get("kv_from")))
        x = x + y + (_gelu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
    return norm(x[-1:], w["final.norm"]) @ w["head"].T


def exact(case, seed):
    """The logits behind every request's last token, whole sequences at once."""
    c = _config(case["model"])
    w = {k: v.to(F64) for k, v in _weights(case, seed).items()}
    logits = _lfm2_logits if case["model"].startswith("lfm2") else _metanex_logits if case["model"].startswith("metanex") else _rofulorn_logits
    steps, ends = _plan(case)
    out = [logits(c, w, torch.tensor(t, device=DEVICE))[0] for t in _tokens(case, seed)]
    kept = []
    for step in steps:
        if any(a + n == ends[i] for i, a, n, _ in step):
            kept.append(torch.stack([out[i] for i, _, _, want in step if want]))
    return kept
