"""What is timed to judge the speed of this engine: twelve passes through its step function, from one decoded token to
the largest prompt, and random ones of the same ranges.

A case is plain values:

* ``model``: one of the shapes that bench.py measures (``0.5b``, ``1.5b``, ``7b``: Qwen2.5) or ``dibulix`` (its 2k sizes);
* ``dtype``: the engine's compute type;
* ``batch`` requests, each over about ``context`` tokens that are in the cache already (whole pages, as a conversation's
  earlier turns are; ``ragged`` spreads them from a half of that to all of it);
* ``first``: the tokens the first request adds, ``new``: the most that each other request adds (from 1 on, ragged);
* ``steps``: how many tokens each request decodes after that, one step each.

A pass admits the requests, lets them share their cached pages, runs the step (or, for a prompt longer than a step may
be, the steps) with the new tokens, decodes, and gives everything back.  The tokens are given, as trace replay gives
them, and the result is the last step's logits: a sampled token may turn on a tie, which no tolerance covers.  Routed
feed-forwards are left out for the same reason: reduced precision may choose another expert where two score alike.
Each step's sampling kernels run as they do when the engine serves."""
import math

import numpy as np
import torch

QWEN2 = {
    "0.5b": dict(num_hidden_layers=24, hidden_size=896, num_attention_heads=14, num_key_value_heads=2, head_dim=64, intermediate_size=4864, vocab_size=151936, tie_word_embeddings=True),
    "1.5b": dict(num_hidden_layers=28, hidden_size=1536, num_attention_heads=12, num_key_value_heads=2, head_dim=128, intermediate_size=8960, vocab_size=151936, tie_word_embeddings=True),
    "7b": dict(num_hidden_layers=28, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4, head_dim=128, intermediate_size=18944, vocab_size=152064, tie_word_embeddings=False),
}
EPS, THETA = 1e-6, 1e6
# Four layers as bench.py has them: delta rule, latent attention, attention beside a minGRU, delta rule.
DIBULIX = dict(width=2048, heads=16, dim=128, rot=64, vdim=128, kv_rank=512, ff=8192, vocab=32000, streams=4, delta_heads=8, delta_kv_heads=4, delta_dim=128, delta_vdim=256, conv=4, low_rank=16,
               kv_heads=4, att_dim=128, att_rot=64, window=1024, gru=4096, kinds=("delta", "latent", "parallel", "delta"))
SCALING = {"factor": 8.0, "original": 2048, "fast": 32.0, "slow": 1.0}
PAGE, STEP_TOKENS, CONTEXT = 64, 2048, 4096


def case(name, model, dtype="bfloat16", batch=1, context=0, ragged=False, first=1, new=1, steps=0):
    c = {"model": model, "dtype": dtype, "batch": batch, "context": context, "ragged": ragged, "first": first, "new": new, "steps": steps}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user, a short conversation: nothing but the latency of a decode step
        case("decode_05b_1", "0.5b", context=128, steps=7),
        # the benchmark's headline: eight requests with 2,048 tokens each
        case("decode_05b_8", "0.5b", batch=8, context=2048, steps=7),
        # a server's full batch
        case("decode_05b_64", "0.5b", batch=64, context=2048, ragged=True, steps=3),
        # an ordinary batch of conversations of different lengths
        case("decode_15b_27", "1.5b", batch=27, context=1536, ragged=True, steps=3),
        # the largest model, where a step is its weights
        case("decode_7b_4", "7b", batch=4, context=1024, ragged=True, steps=3),
        # the time to the first token of a short question
        case("prompt_05b_50", "0.5b", first=50),
        # the benchmark's prompt
        case("prompt_05b_2048", "0.5b", first=2048),
        # a document, taken in portions, each over what the cache holds by then
        case("prompt_15b_5001", "1.5b", first=5001),
        # the largest: a long prompt of the largest model
        case("prompt_7b_1999", "7b", first=1999),
        # a server's step: a portion of one prompt beside the tokens of 32 requests that decode
        case("mixed_15b_500", "1.5b", batch=33, context=768, ragged=True, first=500),
        # a question and its answer in 32 bits, the type the reference computes in
        case("float32_05b_40", "0.5b", dtype="float32", first=40, steps=7),
        # recurrent and latent mixers over several residual streams: whole requests, prompts and decoding
        case("dibulix_4x300", "dibulix", batch=4, first=300, new=300, steps=15),
    ]


def log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prompt", "prompt", "mixed", "float32", "dibulix"))
    if kind == "decode":
        model = rng.choice(("0.5b", "0.5b", "1.5b", "7b"))
        return case(None, model, batch=log_between(rng, 1, 12 if model == "7b" else 64), context=64 * log_between(rng, 1, 16 if model == "7b" else 40), ragged=rng.random() < 0.5,
                    steps=rng.choice((1, 3, 7) if model == "7b" else (3, 7)))
    if kind == "prompt":
        model = rng.choice(("0.5b", "0.5b", "1.5b", "7b"))
        batch = rng.choice((1, 1, 1, log_between(rng, 2, 16)))
        total = log_between(rng, 20, 1999 if model == "7b" else 2048 if batch > 1 else 6000)
        return case(None, model, batch=batch, context=64 * rng.choice((0, 0, 0, 1, 5, 16)), first=max(1, total // batch), new=max(1, total // batch))
    if kind == "mixed":
        model = rng.choice(("0.5b", "1.5b"))
        return case(None, model, batch=log_between(rng, 2, 64), context=64 * log_between(rng, 1, 24), ragged=True, first=log_between(rng, 16, 2048), steps=rng.choice((0, 0, 1)))
    if kind == "float32":
        return case(None, "0.5b", dtype="float32", batch=rng.choice((1, 1, 2, 4)), context=64 * rng.choice((0, 1, 4)), first=log_between(rng, 1, 64), new=8, steps=rng.choice((1, 3, 7)))
    n = log_between(rng, 20, 1200)
    batch = log_between(rng, 1, min(16, 2048 // n))
    return case(None, "dibulix", batch=batch, first=n, new=n, steps=rng.choice((0, 3, 15)))


# ---- what a case's seed decides -------------------------------------------------------------------------------------


def shapes(model):
    """Every tensor of a model: name -> (shape, law)."""
    out = {}
    if model in QWEN2:
        z = QWEN2[model]
        h, q, kv, f = z["hidden_size"], z["num_attention_heads"] * z["head_dim"], z["num_key_value_heads"] * z["head_dim"], z["intermediate_size"]
        out["model.embed_tokens.weight"] = ((z["vocab_size"], h), "embedding")
        for i in range(z["num_hidden_layers"]):
            p = "model.layers.%d." % i
            for n, rows in (("q", q), ("k", kv), ("v", kv)):
                out[p + "self_attn.%s_proj.weight" % n] = ((rows, h), "normal")
                out[p + "self_attn.%s_proj.bias" % n] = ((rows,), "normal")
            out[p + "mlp.gate_proj.weight"] = out[p + "mlp.up_proj.weight"] = ((f, h), "normal")
            out[p + "self_attn.o_proj.weight"], out[p + "mlp.down_proj.weight"] = ((h, q), "residual"), ((h, f), "residual")
            out[p + "input_layernorm.weight"] = out[p + "post_attention_layernorm.weight"] = ((h,), "ones")
        out["model.norm.weight"] = ((h,), "ones")
        if not z["tie_word_embeddings"]:
            out["lm_head.weight"] = ((z["vocab_size"], h), "normal")
        return out
    z = DIBULIX
    w, s = z["width"], z["streams"]
    out["embed"] = ((z["vocab"], w), "normal")
    for i, kind in enumerate(z["kinds"]):
        p = "l%d." % i
        if kind == "delta":
            qk, v, d, r = z["delta_kv_heads"] * z["delta_dim"], z["delta_heads"] * z["delta_vdim"], z["delta_heads"] * z["delta_dim"], z["low_rank"]
            for n, rows in (("q", qk), ("k", qk), ("v", v)):
                out[p + "mix." + n] = ((rows, w), "normal")
                out[p + "mix.%s.conv" % n] = ((rows, z["conv"]), "normal")
            for n, shape in (("b", (z["delta_heads"], w)), ("A_log", (z["delta_heads"],)), ("dt_bias", (d,)), ("o", (w, v)), ("a1", (r, w)), ("a2", (d, r)), ("g1", (r, w)), ("g2", (v, r))):
                out[p + "mix." + n] = (shape, "normal")
            out[p + "mix.norm"] = ((z["delta_vdim"],), "ones")
        elif kind == "latent":
            hh = z["heads"]
            for n, shape in (("uk", (hh * z["dim"], z["kv_rank"])), ("uv", (hh * z["vdim"], z["kv_rank"])), ("o", (w, hh * z["vdim"])), ("dkv", (z["kv_rank"] + z["rot"], w)),
                             ("q", (hh * (z["dim"] + z["rot"]), w)), ("g", (hh, w))):
                out[p + "mix." + n] = (shape, "normal")
            out[p + "mix.dkv.norm"] = ((z["kv_rank"],), "ones")
        else:
            for n, heads in (("q", z["heads"]), ("k", z["kv_heads"]), ("v", z["kv_heads"])):
                out[p + "mix.left." + n] = ((heads * z["att_dim"], w), "normal")
                out[p + "mix.left.%s.b" % n] = ((heads * z["att_dim"],), "normal")
            out[p + "mix.left.o"] = ((w, z["heads"] * z["att_dim"]), "normal")
            for n in ("z", "x", "g"):
                out[p + "mix.right." + n] = ((z["gru"], w), "normal")
            out[p + "mix.right.z.b"] = out[p + "mix.right.x.b"] = ((z["gru"],), "normal")
            out[p + "mix.right.o"] = ((w, z["gru"]), "normal")
        out[p + "mlp.up"], out[p + "mlp.down"] = ((z["ff"], w), "normal"), ((w, z["ff"]), "normal")
        for k in (1, 2):
            out[p + "norm%d" % k] = ((w,), "ones")
            out[p + "hc%d.in" % k] = out[p + "hc%d.out" % k] = ((s,), "ones")
            out[p + "hc%d.mix" % k] = ((s, s), "identity")
    out["final.norm"] = ((w,), "ones")
    return out


def weights(model, seed):
    """bfloat16 on the GPU, drawn as the engine's own random mode draws them: N(0, 0.02), norms near 1.  In Qwen2 models the
    products into the residual stream are narrower by the root of their number, as models start their training, and the
    embedding is N(0, 1), as torch.nn.Embedding's: with 0.02 throughout, 28 layers 3,584 wide multiply a rounding until
    two correct implementations are 4% apart."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    scale = {"normal": 0.02, "embedding": 1.0, "residual": 0.02 / math.sqrt(2 * QWEN2[model]["num_hidden_layers"]) if model in QWEN2 else 0.0}
    out = {}
    for name, (shape, law) in shapes(model).items():
        x = torch.randn(shape, generator=gen, dtype=torch.bfloat16 if law in scale else torch.float32, device="cuda")
        if law in scale:
            x.mul_(scale[law])
        else:
            x = (x * 0.01 + (1.0 if law == "ones" else torch.eye(shape[0], device="cuda"))).to(torch.bfloat16)
        out[name] = x
    return out


def vocabulary(model):
    return QWEN2[model]["vocab_size"] if model in QWEN2 else DIBULIX["vocab"]


def tokens(c, seed):
    """Per request: (tokens in the cache, new tokens, tokens decoded after them)."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(c["batch"]):
        pages = c["context"] // PAGE
        if c["ragged"] and pages > 1:
            pages = int(rng.integers((pages + 1) // 2, pages + 1))
        new = c["first"] if i == 0 else int(rng.integers(1, c["new"] + 1))
        ids = rng.integers(0, vocabulary(c["model"]), pages * PAGE + new + c["steps"]).tolist()
        out.append((ids[: pages * PAGE], ids[pages * PAGE : pages * PAGE + new], ids[pages * PAGE + new :]))
    return out


# ---- the pass ---------------------------------------------------------------------------------------------------------


def build(model):
    """(architecture's description, for the engine) of a model."""
    if model in QWEN2:
        from alofa_b200.models.qwen2 import Qwen2Config, build_spec

        return build_spec(Qwen2Config(rms_norm_eps=EPS, rope_theta=THETA, max_position_embeddings=32768, **QWEN2[model]))
    from alofa_b200.models.dibulix import DeltaConfig, DibulixConfig, DibulixLayer, LatentConfig, ParallelConfig, Rotary, WindowedAttentionConfig, build_spec

    z = DIBULIX
    mixers = {
        "delta": ("channel_delta", DeltaConfig(z["delta_heads"], z["delta_kv_heads"], z["delta_dim"], z["delta_vdim"], z["conv"])),
        "latent": ("latent_attention", LatentConfig(z["heads"], z["dim"], z["rot"], z["vdim"], z["kv_rank"], (z["dim"] + z["rot"]) ** -0.5, Rotary(1e4, z["rot"], dict(SCALING)), z["window"])),
        "parallel": ("parallel", ParallelConfig(WindowedAttentionConfig(z["heads"], z["kv_heads"], z["att_dim"], z["att_dim"], z["att_dim"] ** -0.5, Rotary(1e6, z["att_rot"]), z["window"]),
                                                z["gru"], 1.0, 1.0)),
    }
    return build_spec(DibulixConfig(z["vocab"], z["width"], EPS, 1.0, z["streams"], [DibulixLayer(*mixers[k], z["ff"]) for k in z["kinds"]]))


def prepare(case, seed):
    """A model with its weights, a step runner, and the requests' earlier tokens in its cache."""
    from alofa_b200.engine.loading import compute_dtype
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    model = Model(build(case["model"]), Runtime(torch.device("cuda"), compute_dtype(case["dtype"])))
    model.load(load_state(model.tensors(), weights(case["model"], seed), model.rt.dtype, model.rt.device))
    requests = tokens(case, seed)
    longest = max(len(a) + len(b) + len(d) for a, b, d in requests)
    pages = sum(len(a) // PAGE + 2 + (len(b) + len(d)) // PAGE for a, b, d in requests)
    runner = StepRunner(model, block_size=PAGE, num_pages=pages, max_requests=2 * case["batch"], max_tokens=max(CONTEXT, -(-longest // PAGE) * PAGE),
                        max_step_tokens=STEP_TOKENS + case["batch"])
    sources = []
    for i, (cached, _, _) in enumerate(requests):
        if cached:
            sources.append(runner.admit(1_000_000 + i))
            for lo in range(0, len(cached), STEP_TOKENS):
                runner.forward([StepEntry(sources[-1], cached[lo : lo + STEP_TOKENS])])
    runner.check_status()
    return {"runner": runner, "sources": sources, "cached": [len(a) for a, _, _ in requests], "new": [b for _, b, _ in requests], "decoded": [d for _, _, d in requests]}


def run(state):
    from alofa_b200.engine.step import StepEntry

    runner, new = state["runner"], state["new"]
    slots = [runner.admit(i) for i in range(len(new))]
    for slot, source, n in zip(slots, state["sources"], state["cached"]):
        runner.manager.share_prefix(source, slot, n)
    ahead = max(0, -(-len(new[0]) // STEP_TOKENS) - 1) * STEP_TOKENS  # a prompt longer than a step: its portions but the last run alone
    for lo in range(0, ahead, STEP_TOKENS):
        runner.forward([StepEntry(slots[0], new[0][lo : lo + STEP_TOKENS])])
    entries = [StepEntry(s, ids[ahead:] if i == 0 else ids, (len(ids) - (ahead if i == 0 else 0) - 1,)) for i, (s, ids) in enumerate(zip(slots, new))]
    _, logits, _ = runner.forward_sampled(entries)
    for t in range(len(state["decoded"][0])):
        _, logits, _ = runner.forward_sampled([StepEntry(s, ids[t : t + 1], (0,)) for s, ids in zip(slots, state["decoded"])])
    for slot in slots:
        runner.release(slot)
    return logits


# ---- what it costs at the least, and what it should give ---------------------------------------------------------------


def sizes(model):
    """(numbers in the layers' weights, in the head's, cache numbers a token has, the most tokens a cache keeps, numbers of
    fp32 state a request has, multiply-adds a (query, key) pair takes, width)."""
    inner = sum(math.prod(s) for n, (s, _) in shapes(model).items() if n not in ("model.embed_tokens.weight", "lm_head.weight", "embed"))
    if model in QWEN2:
        z = QWEN2[model]
        return (inner, z["vocab_size"] * z["hidden_size"], z["num_hidden_layers"] * 2 * z["num_key_value_heads"] * z["head_dim"], 1 << 30, 0,
                z["num_hidden_layers"] * 2 * z["num_attention_heads"] * z["head_dim"], z["hidden_size"])
    z = DIBULIX
    row, kv = z["kv_rank"] + z["rot"], 2 * z["kv_heads"] * z["att_dim"]
    delta_state = z["delta_heads"] * z["delta_dim"] * z["delta_vdim"] + (z["conv"] - 1) * (2 * z["delta_kv_heads"] * z["delta_dim"] + z["delta_heads"] * z["delta_vdim"])
    return (inner, z["vocab"] * z["width"], row + kv, z["window"], 2 * delta_state + z["gru"], z["heads"] * (z["dim"] + z["rot"] + z["vdim"]) + 2 * z["heads"] * z["att_dim"], z["width"])


def work(case):
    """Per step: every weight and the cached rows of the step's requests read once, new rows and wanted logits written;
    multiply-adds of every token through the weights and with every key it sees."""
    inner, head, row, kept, state, pair, width = sizes(case["model"])
    size = 4 if case["dtype"] == "float32" else 2
    total_bytes = total_flops = 0
    requests = tokens(case, 0)
    ahead = max(0, -(-case["first"] // STEP_TOKENS) - 1)
    passes = [[(k * STEP_TOKENS, STEP_TOKENS)] for k in range(ahead)]
    passes.append([(len(a) + (ahead * STEP_TOKENS if i == 0 else 0), len(b) - (ahead * STEP_TOKENS if i == 0 else 0)) for i, (a, b, _) in enumerate(requests)])
    passes += [[(len(a) + len(b) + t, 1) for a, b, _ in requests] for t in range(case["steps"])]
    for k, step in enumerate(passes):
        rows = sum(n for _, n in step)
        wanted = len(step) if k >= ahead else 0
        total_bytes += size * (inner + (head if wanted else 0) + rows * width + row * (rows + sum(min(have, kept) for have, _ in step))) + 4 * wanted * vocabulary(case["model"]) + 8 * state * len(step)
        total_flops += 2 * (rows * inner + wanted * head + pair * sum(sum(min(have + j + 1, kept) for j in range(n)) for have, n in step))
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    # measured against exact(): 6e-7 to 1e-6 in 32 bits; in bfloat16 0.0018 (0.5b), 0.0022 (1.5b), 0.0054 (7b), 0.0056 (dibulix)
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 5e-5}
    return {"rel": 2e-2, "max": 1.5e-1}


def rms(x, weight):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * weight


def attend(q, k, v, scale, window=None, one_more=False):
    """q [T, H, d], k [T, G, d], v [T, G, e] -> [T, H e], every position over those up to it (the last `window` of them)."""
    n, heads, group = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    at = torch.arange(n, device=q.device)
    hidden = at[None, :] > at[:, None]
    if window:
        hidden |= at[None, :] <= at[:, None] - window
    out = []
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].T * scale).masked_fill_(hidden, -math.inf)
        top = s.amax(-1, keepdim=True)
        e = s.sub_(top).exp_()
        out.append(e @ v[:, h // group] / (e.sum(-1, keepdim=True) + (torch.exp(-top) if one_more else 0.0)))
    return torch.cat(out, -1)


def turned(x, cos, sin, pairs=False):
    """x [T, heads, d]: its first 2 * cos.shape[-1] numbers a head turned, neighbours together or one half with the other."""
    d = 2 * cos.shape[-1]
    c, s = cos[:, None], sin[:, None]
    a, b = (x[..., 0:d:2], x[..., 1:d:2]) if pairs else (x[..., : d // 2], x[..., d // 2 : d])
    out = x.clone()
    if pairs:
        out[..., 0:d:2], out[..., 1:d:2] = a * c - b * s, b * c + a * s
    else:
        out[..., : d // 2], out[..., d // 2 : d] = a * c - b * s, b * c + a * s
    return out


def qwen2_rows(ids, w, z):
    n, heads, groups, d = len(ids), z["num_attention_heads"], z["num_key_value_heads"], z["head_dim"]
    # frequencies and angles are 32-bit numbers by definition
    inv = np.float32(1.0) / np.power(np.float64(THETA), 2.0 * np.arange(d // 2) / d).astype(np.float32)
    angle = torch.from_numpy((np.arange(n, dtype=np.float32)[:, None] * inv[None, :]).astype(np.float64)).cuda()
    cos, sin = angle.cos(), angle.sin()
    x = w["model.embed_tokens.weight"][torch.tensor(ids, device="cuda")]
    for i in range(z["num_hidden_layers"]):
        p = "model.layers.%d." % i
        y = rms(x, w[p + "input_layernorm.weight"])
        q, k, v = ((y @ w[p + "self_attn.%s_proj.weight" % m].T + w[p + "self_attn.%s_proj.bias" % m]).view(n, -1, d) for m in "qkv")
        x = x + attend(turned(q, cos, sin), turned(k, cos, sin), v, d**-0.5) @ w[p + "self_attn.o_proj.weight"].T
        y = rms(x, w[p + "post_attention_layernorm.weight"])
        x = x + (torch.nn.functional.silu(y @ w[p + "mlp.gate_proj.weight"].T) * (y @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return rms(x[-1], w["model.norm.weight"])


def stretched(dims, base):
    """Frequencies between themselves and an eighth of themselves along a ramp over the pairs, and the factor on the turn."""
    i = torch.arange(dims // 2, dtype=torch.float64)
    f = base ** (-2.0 * i / dims)
    place = lambda turns: dims * math.log(SCALING["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(place(SCALING["fast"])), 0), min(math.ceil(place(SCALING["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / SCALING["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(SCALING["factor"]) + 1.0


def delta_mixer(y, w, p, z):
    n, heads, groups, d, dv = len(y), z["delta_heads"], z["delta_kv_heads"], z["delta_dim"], z["delta_vdim"]

    def convolved(name):
        u, taps = y @ w[p + name].T, w[p + name + ".conv"]
        u = torch.cat([u.new_zeros(taps.shape[1] - 1, u.shape[1]), u])
        return torch.nn.functional.silu(sum(u[t : t + n] * taps[:, t] for t in range(taps.shape[1])))

    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = (unit(convolved("q").view(n, groups, d)) * d**-0.5).repeat_interleave(heads // groups, 1)
    k = unit(convolved("k").view(n, groups, d)).repeat_interleave(heads // groups, 1)
    v, beta = convolved("v").view(n, heads, dv), torch.sigmoid(y @ w[p + "b"].T)
    decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * torch.nn.functional.softplus((y @ w[p + "a1"].T @ w[p + "a2"].T + w[p + "dt_bias"]).view(n, heads, d)))
    state, out = y.new_zeros(heads, d, dv), []
    for t in range(n):
        state = state * decay[t][:, :, None]
        state = state + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hd,hde->he", k[t], state)))[:, None, :]
        out.append(torch.einsum("hd,hde->he", q[t], state))
    o = rms(torch.stack(out), w[p + "norm"]) * torch.sigmoid(y @ w[p + "g1"].T @ w[p + "g2"].T).view(n, heads, dv)
    return o.reshape(n, -1) @ w[p + "o"].T


def latent_mixer(y, w, p, z):
    n, heads, d, r, rank = len(y), z["heads"], z["dim"], z["rot"], z["kv_rank"]
    f, factor = stretched(r, 1e4)
    angle = (torch.arange(n, dtype=torch.float64)[:, None] * f).cuda()
    cos, sin = angle.cos() * factor, angle.sin() * factor
    q, low = (y @ w[p + "q"].T).view(n, heads, d + r), y @ w[p + "dkv"].T
    c = rms(low[:, :rank], w[p + "dkv.norm"])
    q = torch.cat([q[..., :d], turned(q[..., d:], cos, sin)], -1)
    k = torch.cat([(c @ w[p + "uk"].T).view(n, heads, d), turned(low[:, rank:].reshape(n, 1, r), cos, sin).expand(n, heads, r)], -1)
    o = attend(q, k, (c @ w[p + "uv"].T).view(n, heads, -1), (d + r) ** -0.5, z["window"])
    return (o.view(n, heads, -1) * torch.sigmoid(y @ w[p + "g"].T)[:, :, None]).reshape(n, -1) @ w[p + "o"].T


def parallel_mixer(y, w, p, z):
    n, d = len(y), z["att_dim"]
    angle = (torch.arange(n, dtype=torch.float64)[:, None] * 1e6 ** (-torch.arange(0, z["att_rot"], 2, dtype=torch.float64) / z["att_rot"])).cuda()
    q, k, v = ((y @ w[p + "left." + m].T + w[p + "left.%s.b" % m]).view(n, -1, d) for m in "qkv")
    left = attend(turned(q, angle.cos(), angle.sin(), True), turned(k, angle.cos(), angle.sin(), True), v, d**-0.5, z["window"], one_more=True) @ w[p + "left.o"].T
    move, u = torch.sigmoid(y @ w[p + "right.z"].T + w[p + "right.z.b"]), y @ w[p + "right.x"].T + w[p + "right.x.b"]
    goal = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
    state, out = torch.zeros_like(u[0]), []
    for t in range(n):
        state = state + move[t] * (goal[t] - state)
        out.append(state)
    return left + (torch.stack(out) * torch.nn.functional.silu(y @ w[p + "right.g"].T)) @ w[p + "right.o"].T


def dibulix_rows(ids, w, z):
    x = w["embed"][torch.tensor(ids, device="cuda")]
    streams = torch.stack([x] * z["streams"])
    mixers = {"delta": delta_mixer, "latent": latent_mixer, "parallel": parallel_mixer}
    for i, kind in enumerate(z["kinds"]):
        p = "l%d." % i
        for k, part in ((1, lambda y: mixers[kind](y, w, p + "mix.", z)), (2, lambda y: torch.relu(y @ w[p + "mlp.up"].T).square() @ w[p + "mlp.down"].T)):
            hc = p + "hc%d." % k
            y = part(rms(torch.einsum("s,sne->ne", w[hc + "in"], streams), w[p + "norm%d" % k]))
            streams = torch.einsum("st,sne->tne", w[hc + "mix"], streams) + w[hc + "out"][:, None, None] * y
    return rms(streams.sum(0)[-1], w["final.norm"])


def exact(case, seed):
    """The last step's logits in 64 bits: each request's whole sequence at once, without a cache."""
    if work(case)["flops"] + 2 * sum(len(a) for a, _, _ in tokens(case, seed)) * sizes(case["model"])[0] > 2.5e14:
        return None
    w = {n: t.double() for n, t in weights(case["model"], seed).items()}
    z, rows = (QWEN2[case["model"]], qwen2_rows) if case["model"] in QWEN2 else (DIBULIX, dibulix_rows)
    last = torch.stack([rows(a + b + d, w, z) for a, b, d in tokens(case, seed)])
    head = w["lm_head.weight" if "lm_head.weight" in w else "embed" if "embed" in w else "model.embed_tokens.weight"]
    return last @ head.T
