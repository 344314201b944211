"""The work that this engine is measured on: requests served through its step function.

A case is a number of requests with prompts of some length and some tokens that follow each
prompt. One pass opens the requests, runs their prompts in portions as the scheduler cuts them
(at most 2,048 tokens of a request and 4,096 tokens a step, running decodes first), then feeds one
token a request and step, keeps the 32-bit logits of every prompt's end and of every token that
follows, and closes the requests. The tokens that follow are given and not chosen, as where a text
is scored or a recorded conversation is replayed: which token wins a near tie would otherwise
decide what all later steps compute. With ``every`` > 0 the requests do not start together: one
arrives every so many steps, so that prompts' portions and decodes share steps, as under a server.

Models: LFM2 in its three published sizes, the architecture that the engine is built around, and
Galarax, which stands for the designs with a matrix of state per head (the delta rule) beside
softmax attention. Weights are random, of the distribution that random models have everywhere in
this repository; token ids are uniform. bfloat16 is what a server runs; float32 is the engine's
other execution type, true 32-bit throughout, for checking a model or a text's score.
"""

import math
import random

import torch

VOCAB = 65536
PAGE = 16
PORTION, STEP = 2048, 4096

_KINDS = ["conv", "conv", "full_attention", "conv", "conv", "full_attention", "conv", "conv",
          "full_attention", "conv", "full_attention", "conv", "full_attention", "conv",
          "full_attention", "conv"]


def _lfm2(hidden, heads, ff):
    return dict(model_type="lfm2", num_hidden_layers=16, layer_types=_KINDS, hidden_size=hidden,
                num_attention_heads=heads, num_key_value_heads=8, block_auto_adjust_ff_dim=True,
                block_ff_dim=ff, block_multiple_of=256, block_ffn_dim_multiplier=1.0,
                vocab_size=VOCAB, rope_theta=1000000.0, conv_L_cache=3, conv_bias=False,
                tie_embedding=True, norm_eps=1e-5, max_position_embeddings=128000)


def _galarax(width):
    left = {"heads": width // 64, "kv_heads": width // 256, "dim": 64, "vdim": 64, "scale": 0.125,
            "rot": {"base": 1000000.0, "dims": 32, "scaling": {
                "factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    right = {"heads": width // 128, "kv_heads": width // 256, "dim": 128, "vdim": 128, "conv": 4}
    layer = {"type": "parallel", "mixer": {"left": left, "right": right},
             "mlp": {"kind": "dense", "ff": 4 * width}}
    return {"architecture": "Galarax", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-6},
            "layers": [layer] * 8}


MODELS = {"lfm2-350m": _lfm2(1024, 16, 6656), "lfm2-700m": _lfm2(1536, 24, 10240),
          "lfm2-1.2b": _lfm2(2048, 32, 12288), "galarax-1024": _galarax(1024),
          "galarax-2048": _galarax(2048)}


def _case(model, dtype, requests, prompt, new, every=0, name=None):
    case = dict(model=model, dtype=dtype, requests=requests, prompt=prompt, new=new, every=every)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one short exchange with the smallest model: the published protocol of 128 tokens in and
        # 16 out; bound by launches and by how fast a step follows the one before
        _case("lfm2-350m", "bfloat16", 1, 128, 16, name="reply_350m"),
        # one user's chat turn with the largest: weights streamed for one token a step
        _case("lfm2-1.2b", "bfloat16", 1, 509, 64, name="chat_1200m"),
        # a small server: eight conversations of about 2,048 tokens go on together
        _case("lfm2-1.2b", "bfloat16", 8, 2048, 64, name="batch8_1200m"),
        # a full server: 64 short requests decode together
        _case("lfm2-1.2b", "bfloat16", 64, 96, 32, name="batch64_1200m"),
        # requests that come and go: portions of prompts beside running decodes in most steps
        _case("lfm2-700m", "bfloat16", 24, 400, 40, every=2, name="arrivals_700m"),
        # time to the first token of a prompt of ordinary length, and of a short one
        _case("lfm2-1.2b", "bfloat16", 1, 2048, 0, name="prompt2048_1200m"),
        _case("lfm2-700m", "bfloat16", 1, 333, 0, name="prompt333_700m"),
        # a long document: attention over up to 16,411 keys
        _case("lfm2-350m", "bfloat16", 1, 16411, 0, name="prompt16411_350m"),
        # the 32-bit engine: the same short exchange, and a few prompts of ordinary length scored
        _case("lfm2-350m", "float32", 1, 128, 16, name="reply_350m_f32"),
        _case("lfm2-1.2b", "float32", 4, 300, 8, name="batch4_1200m_f32"),
        # the delta rule: a prompt (the recurrence over 2,048 tokens), and eight requests that decode
        _case("galarax-2048", "bfloat16", 1, 2048, 0, name="prompt2048_galarax"),
        _case("galarax-1024", "bfloat16", 8, 160, 48, name="batch8_galarax"),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _cost(case):
    """A rough time of a pass, to keep drawn cases within the listed ones."""
    need = work(case)
    return need["bytes"] / 4e12 + need["flops"] / (8e14 if case["dtype"] == "bfloat16" else 1e13)


def draw(rng):
    most = {kind: max(_cost(c) for c in listed() if c["dtype"] == kind)
            for kind in ("bfloat16", "float32")}
    while True:
        dtype = rng.choice(["bfloat16"] * 4 + ["float32"])
        models = list(MODELS) if dtype == "bfloat16" else ["lfm2-350m", "lfm2-700m", "lfm2-1.2b"]
        requests = _spread(rng, 1, 64)
        case = _case(rng.choice(models), dtype, requests, _spread(rng, 5, 16411),
                     rng.choice([0, _spread(rng, 1, 64)]),
                     rng.choice([0, 0, 1, 2, 3]) if requests > 1 else 0)
        if _cost(case) <= most[dtype]:
            return case


# ------------------------------------------------------------------ the shape of a pass


def _lengths(case):
    """The prompts' lengths: between three quarters and five quarters of the case's, the same for
    every seed; a single prompt has the length that the case names."""
    if case["requests"] == 1:
        return [case["prompt"]]
    rng = random.Random("%d of %d" % (case["requests"], case["prompt"]))
    return [max(1, round(case["prompt"] * rng.uniform(0.75, 1.25)))
            for _ in range(case["requests"])]


def _steps(case):
    """The pass step by step: lists of (request, first token, end, whether its last token's logits
    are kept), decodes ahead of portions."""
    lengths, new, every = _lengths(case), case["new"], case["every"]
    done = [0] * len(lengths)
    steps = []
    while any(d < n + new for d, n in zip(done, lengths)):
        here = len(lengths) if every == 0 else min(len(lengths), len(steps) // every + 1)
        step, room = [], STEP
        for r in range(here):
            if lengths[r] <= done[r] < lengths[r] + new:
                step.append((r, done[r], done[r] + 1, True))
                room -= 1
        for r in range(here):
            if done[r] < lengths[r] and room > 0:
                end = min(lengths[r], done[r] + PORTION, done[r] + room)
                step.append((r, done[r], end, end == lengths[r]))
                room -= end - done[r]
        for r, _, end, _ in step:
            done[r] = end
        if step or every:
            steps.append(step)
    return [s for s in steps if s]


def _described(case):
    from mlx_one_b200.config import architecture_key, get_architecture

    data = MODELS[case["model"]]
    architecture = get_architecture(architecture_key(data))
    config = architecture.config_class.from_dict(data)
    return architecture, config, architecture.describe(config)


def _tensors(case, spec, seed):
    from mlx_one_b200.weights import random_tensors

    tensors = random_tensors(spec, seed=seed, dtype=getattr(torch, case["dtype"]), device="cuda:0")
    # Rows of the embedding with values around one, so that a token is still seen behind the first
    # layers, as in a trained model. With 0.02 everywhere the first outputs drown it, and 16-bit
    # roundings grow from layer to layer: two correct products then differ by 2 % at the logits.
    for name in ("model.embed_tokens.weight", "embed"):
        if name in tensors:
            tensors[name] *= 50.0
    return tensors


def _tokens(case, seed):
    rng = torch.Generator().manual_seed(1000003 * seed + 17)
    return [torch.randint(0, VOCAB, (n + case["new"],), generator=rng).tolist()
            for n in _lengths(case)]


def _rows(case):
    return sum(keep for step in _steps(case) for *_, keep in step)


# ------------------------------------------------------------------ one pass


def prepare(case, seed):
    """A loaded model with its engine, the requests' token ids, and room for the logits."""
    from pathlib import Path

    from mlx_one_b200 import BatchingConfig, CacheConfig, Engine
    from mlx_one_b200.engine.loading import LoadedModel, build_model
    from mlx_one_b200.engine.runner import StepEntry

    architecture, config, spec = _described(case)
    model = build_model(spec, _tensors(case, spec, seed), case["dtype"], "cuda:0")
    requests = case["requests"]
    capacity = sum(-(-(n + case["new"]) // PAGE) * PAGE for n in _lengths(case))
    engine = Engine(LoadedModel(Path("random"), architecture, config, spec, model),
                    execution_dtype=case["dtype"],
                    batching_config=BatchingConfig(max_sequences=requests,
                                                   queue_size=requests + 1,
                                                   prefill_chunk_size=PORTION,
                                                   max_scheduled_tokens=STEP,
                                                   max_prefill_tokens=STEP),
                    cache_config=CacheConfig(block_size_tokens=PAGE, capacity_tokens=capacity,
                                             max_requests=requests))
    tokens = _tokens(case, seed)
    plan = [[StepEntry(r, tokens[r][first:end], (end - first - 1,) if keep else ())
             for r, first, end, keep in step] for step in _steps(case)]
    logits = torch.empty((_rows(case), VOCAB), dtype=torch.float32, device="cuda:0")
    return {"engine": engine, "plan": plan, "logits": logits, "requests": requests}


def run(state):
    engine, logits = state["engine"], state["logits"]
    for r in range(state["requests"]):
        engine.cache.open(r)
    at = 0
    for entries in state["plan"]:
        got = engine.runner.step(entries)
        if got is not None:
            logits[at:at + got.shape[0]].copy_(got)
            at += got.shape[0]
    for r in range(state["requests"]):
        engine.cache.close(r)
    return logits


# ------------------------------------------------------------------ what a pass needs


def _parameters(case):
    """(values of all matrices that a token passes but the table and the head, softmax heads' width,
    keys' width, layers with softmax attention, values of recurrent state of a request)."""
    data = MODELS[case["model"]]
    if "model_type" in data:
        width = data["hidden_size"]
        ff = -(-int(2 * data["block_ff_dim"] / 3) // 256) * 256
        keys = 8 * (width // data["num_attention_heads"])
        attention = _KINDS.count("full_attention")
        conv = len(_KINDS) - attention
        values = len(_KINDS) * 3 * width * ff + conv * 4 * width * width + \
            attention * (2 * width * width + 2 * width * keys)
        return width, values, width, keys, attention, conv * 2 * width
    width, left, right = data["width"], data["layers"][0]["mixer"]["left"], \
        data["layers"][0]["mixer"]["right"]
    keys, inner = left["kv_heads"] * left["dim"], right["heads"] * right["vdim"]
    per = 2 * width * width + 2 * width * keys + 3 * width * inner + \
        2 * width * right["kv_heads"] * right["dim"] + 2 * width * right["heads"] + 8 * width * width
    layers = len(data["layers"])
    return width, layers * per, width, keys, layers, layers * inner * right["dim"]


def work(case):
    """Every step reads the weights once (the head's where it gives logits), its requests' keys,
    values and state, and writes what it adds to them and its logits."""
    width, values, inner, keys, attention, state = _parameters(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    bytes_, flops = 0.0, 0.0
    for step in _steps(case):
        rows = sum(keep for *_, keep in step)
        bytes_ += size * (values + (VOCAB * width if rows else 0)) + 4 * rows * VOCAB
        flops += 2.0 * rows * VOCAB * width
        for _, first, end, _ in step:
            tokens = end - first
            bytes_ += size * (tokens * width + 2 * keys * attention * (end + tokens)) + 8 * state
            flops += tokens * (2.0 * values + 3 * state)
            flops += 4.0 * inner * attention * (tokens * first + tokens * (tokens + 1) / 2)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """bfloat16: with the library's products in the place of this engine's (another order of
    additions, one rounding more behind a gate) the logits move by 0.4 to 1.4 %, single ones by up to
    8 % of their root mean square; the engine itself is 1 to 1.2 % from 64 bits. float32: 1e-5 from
    64 bits."""
    if case["dtype"] == "float32":
        return {"rel": 4e-5, "max": 4e-4}
    return {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------ the same in 64 bits


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(count, frequencies):
    """Positions times frequencies, in 32-bit as the models define them."""
    at = torch.arange(count, dtype=torch.float32, device="cuda:0")
    return (at[:, None] * frequencies.to("cuda:0", torch.float32)[None, :]).double()[:, None, :]


def _turn(x, angles, amplitude=1.0):
    half = angles.shape[-1]
    a, b, rest = x[..., :half], x[..., half:2 * half], x[..., 2 * half:]
    cos, sin = torch.cos(angles) * amplitude, torch.sin(angles) * amplitude
    return torch.cat((a * cos - b * sin, b * cos + a * sin, rest), -1)


def _attend(q, k, v, scale):
    """q [T, H, D], k and v [T, G, D]: causal softmax attention, 1,024 queries at a time."""
    count, heads, _ = q.shape
    group = heads // k.shape[1]
    out = torch.empty_like(q)
    for h in range(heads):
        for at in range(0, count, 1024):
            end = min(count, at + 1024)
            s = (q[at:end, h] @ k[:end, h // group].T) * scale
            hidden = torch.arange(end, device=s.device)[None, :] > \
                torch.arange(at, end, device=s.device)[:, None]
            out[at:end, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ \
                v[:end, h // group]
    return out


def _causal_conv(x, w):
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * w[:, j] for j in range(taps))


def _lfm2_stream(data, w, ids):
    eps, heads = data["norm_eps"], data["num_attention_heads"]
    width, count = data["hidden_size"], len(ids)
    dim = width // heads
    x = w("model.embed_tokens.weight")[ids]
    half = dim // 2
    turns = torch.pow(torch.tensor(data["rope_theta"]), -torch.arange(half).float() / half)
    for i, kind in enumerate(_KINDS):
        p = f"model.layers.{i}."
        n = _rms(x, eps) * w(p + "operator_norm.weight")
        if kind == "conv":
            b, c, u = (n @ w(p + "conv.in_proj.weight").T).chunk(3, -1)
            x = x + (c * _causal_conv(b * u, w(p + "conv.conv"))) @ w(p + "conv.out_proj.weight").T
        else:
            p += "self_attn."
            q = (n @ w(p + "q_proj.weight").T).view(count, heads, dim)
            k = (n @ w(p + "k_proj.weight").T).view(count, -1, dim)
            v = (n @ w(p + "v_proj.weight").T).view(count, -1, dim)
            angles = _angles(count, turns)
            q = _turn(_rms(q, eps) * w(p + "q_layernorm.weight"), angles)
            k = _turn(_rms(k, eps) * w(p + "k_layernorm.weight"), angles)
            x = x + _attend(q, k, v, dim ** -0.5).reshape(count, width) @ w(p + "out_proj.weight").T
            p = f"model.layers.{i}."
        n = _rms(x, eps) * w(p + "ffn_norm.weight")
        p += "feed_forward."
        x = x + (torch.nn.functional.silu(n @ w(p + "w1.weight").T) * (n @ w(p + "w3.weight").T)) \
            @ w(p + "w2.weight").T
    return _rms(x, eps) * w("model.embedding_norm.weight")


def _stretched(rot):
    dims, base, s = rot["dims"], rot["base"], rot["scaling"]
    i = torch.arange(dims // 2, dtype=torch.float64)
    f = base ** (-2 * i / dims)

    def at(turns):
        return dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    low, high = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
    ramp = torch.clamp((i - low) / max(high - low, 0.001), 0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1


def _delta(q, k, v, beta, g):
    """S = g S; u = beta (v - S^T k); S = S + k u^T; o = S^T q, all heads side by side."""
    count, heads, _ = v.shape
    group = heads // q.shape[1]
    q, k = q.repeat_interleave(group, 1), k.repeat_interleave(group, 1)
    s = v.new_zeros(heads, q.shape[2], v.shape[2])
    out = torch.empty_like(v)
    for t in range(count):
        s *= g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None, :], s)[:, 0])
        s += k[t, :, :, None] * u[:, None, :]
        out[t] = torch.bmm(q[t, :, None, :], s)[:, 0]
    return out


def _galarax_stream(data, w, ids):
    eps, count = data["norm"]["eps"], len(ids)
    silu = torch.nn.functional.silu
    x = w("embed")[ids]
    for i, layer in enumerate(data["layers"]):
        n = _rms(x, eps) * (1 + w(f"l{i}.norm1"))
        p, c = f"l{i}.mix.left.", layer["mixer"]["left"]
        turns, amplitude = _stretched(c["rot"])
        angles = _angles(count, turns)
        q = (n @ w(p + "q").T + w(p + "q.b")).view(count, c["heads"], c["dim"])
        k = (n @ w(p + "k").T + w(p + "k.b")).view(count, c["kv_heads"], c["dim"])
        v = (n @ w(p + "v").T + w(p + "v.b")).view(count, c["kv_heads"], c["vdim"])
        q, k = _rms(_turn(q, angles, amplitude), eps), _rms(_turn(k, angles, amplitude), eps)
        a = _attend(q, k, v, c["scale"]).reshape(count, -1) @ w(p + "o").T
        a = _rms(a, eps) * w(p + "out")
        p, c = f"l{i}.mix.right.", layer["mixer"]["right"]

        def unit(y):
            return y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)

        q, k, v = (silu(_causal_conv(n @ w(p + z).T, w(p + z + ".conv"))) for z in "qkv")
        q = unit(q.view(count, c["kv_heads"], -1)) * c["dim"] ** -0.5
        k = unit(k.view(count, c["kv_heads"], -1))
        beta = torch.sigmoid(n @ w(p + "b").T)
        g = torch.exp(-torch.exp(w(p + "A_log")) *
                      torch.nn.functional.softplus(n @ w(p + "a").T + w(p + "dt_bias")))
        o = _delta(q, k, v.view(count, c["heads"], -1), beta, g)
        o = _rms(o, eps) * w(p + "norm") * silu(n @ w(p + "g").T).view(count, c["heads"], -1)
        b = o.reshape(count, -1) @ w(p + "o").T
        x = x + 0.5 * (a + _rms(b, eps) * w(p + "out"))
        n = _rms(x, eps) * (1 + w(f"l{i}.norm2"))
        x = x + torch.relu(n @ w(f"l{i}.mlp.up").T) ** 2 @ w(f"l{i}.mlp.down").T
    return _rms(x, eps) * (1 + w("final.norm"))


@torch.no_grad()
def exact(case, seed):
    data = MODELS[case["model"]]
    lfm2 = "model_type" in data
    if not lfm2 and sum(_lengths(case)) + case["requests"] * case["new"] > 20000:
        return None                     # the recurrence runs token by token here
    _, _, spec = _described(case)
    tensors = _tensors(case, spec, seed)
    wide = {name: t.double() for name, t in tensors.items()}
    stream, head = (_lfm2_stream, "model.embed_tokens.weight") if lfm2 else (_galarax_stream, "head")
    logits = torch.empty((_rows(case), VOCAB), dtype=torch.float64, device="cuda:0")
    # the row of each kept (request, token), in the order of the steps
    places = [(r, end - 1) for step in _steps(case) for r, _, end, keep in step if keep]
    for r, ids in enumerate(_tokens(case, seed)):
        mine = [i for i, (owner, _) in enumerate(places) if owner == r]
        x = stream(data, wide.__getitem__, torch.tensor(ids, device="cuda:0"))
        at = torch.tensor([places[i][1] for i in mine], device="cuda:0")
        logits[torch.tensor(mine, device="cuda:0")] = x[at] @ wide[head].T
    return logits
