"""The work whose time counts: whole calls of the Llama decoder (a prompt, and replies to short prompts) and single layers of the
engine's decoders (attention, routed experts, latent attention, recurrences, differential attention) over prompts and in decode steps.

A layer is reached as a model reaches it: a one-layer model is loaded from a configuration and named tensors, the runner lays out the
step (`ModelRunner.prepare`) and the part's `forward(x, ctx, cache)` is the pass.  Single-token steps of a layer run as a captured graph,
since that is how the engine runs every decode step.  Layer sizes are those of the repository's own benchmark configurations.

`exact` is the same arithmetic in float64 on whole sequences, from the same named tensors, in plain torch.
"""
import math
import zlib

import torch

from qorvix_b200.cache.manager import CompositeCacheView
from qorvix_b200.config import lookup_architecture
from qorvix_b200.engine import ModelRunner, StepEntry

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DTYPES = {"bfloat16": BF16, "float32": F32}
EPS = 1e-5
KEY_EPS = 1e-6                     # under the root of the delta rule's unit vectors

MODELS = {
    "1b": dict(architectures=["LlamaForCausalLM"], vocab_size=128256, hidden_size=2048, intermediate_size=8192, num_hidden_layers=16,
               num_attention_heads=32, num_key_value_heads=8, head_dim=64, max_position_embeddings=8192, rms_norm_eps=1e-5,
               rope_theta=500000.0, rope_scaling=dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                                      original_max_position_embeddings=8192), tie_word_embeddings=True),
    "tiny": dict(architectures=["LlamaForCausalLM"], vocab_size=384, hidden_size=192, intermediate_size=512, num_hidden_layers=3,
                 num_attention_heads=6, num_key_value_heads=2, head_dim=32, max_position_embeddings=256, rms_norm_eps=1e-6,
                 rope_theta=500000.0, rope_scaling=dict(rope_type="llama3", factor=8.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                                        original_max_position_embeddings=64), tie_word_embeddings=True),
}

# layer sizes: "large" as the designs are benchmarked, "small" a size below
PARTS = {
    "attention": {"large": dict(width=4096, heads=32, kv=8, dim=128), "small": dict(width=2048, heads=32, kv=8, dim=64)},
    "experts": {"large": dict(width=2048, experts=64, top=6, ff=1408, shared=2816),
                "small": dict(width=1024, experts=32, top=4, ff=704, shared=1408)},
    "latent": {"large": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, rank=512),
               "small": dict(width=1024, heads=8, dim=128, rot=64, vdim=128, rank=256)},
    "mlstm": {"large": dict(width=2048, heads=4, dim=256, vdim=512), "small": dict(width=1024, heads=4, dim=128, vdim=256)},
    "mamba2": {"large": dict(width=2048, heads=64, vdim=64, state=128, taps=4), "small": dict(width=1024, heads=32, vdim=64, state=64, taps=4)},
    "channel_delta": {"large": dict(width=2048, heads=16, kv=8, dim=128, taps=4, rank=64),
                      "small": dict(width=1024, heads=8, kv=8, dim=64, taps=4, rank=32)},
    "diff_attention": {"large": dict(width=2048, heads=16, kv=4, dim=64, vdim=128, window=1024),
                       "small": dict(width=1024, heads=8, kv=4, dim=64, vdim=128, window=512)},
}
STATEFUL = ("mlstm", "mamba2", "channel_delta")
ROT = {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 16.0, "slow": 2.0}}


def _part(name, part, new, past=0, requests=1, size="large", dtype="bfloat16"):
    """`requests` requests that each bring `new` tokens (later ones fewer, down to half) to `past` cached ones (likewise)."""
    return {"name": name, "kind": "part", "part": part, "size": size, "dtype": dtype, "requests": requests, "new": new, "past": past}


def listed():
    return [
        # a prompt of ordinary length through a whole model: what a request's first token waits for
        {"name": "llama_1b_prompt", "kind": "prompt", "model": "1b", "dtype": "bfloat16", "tokens": 2048},
        # eight requests with short prompts, one mixed step and then captured decode steps: a chat server's steady work
        {"name": "llama_1b_replies", "kind": "replies", "model": "1b", "dtype": "bfloat16", "requests": 8, "prompt": 48, "steps": 8},
        # the smallest calls: a tiny model on the 32-bit path, three requests, where launches are all there is
        {"name": "tiny_float32_replies", "kind": "replies", "model": "tiny", "dtype": "float32", "requests": 3, "prompt": 21, "steps": 6},
        # one layer's attention in a decode step of 64 requests with contexts of 1,024 to 2,047 tokens
        _part("attention_decode", "attention", 1, past=2047, requests=64),
        # routed experts over a prompt, and in a decode step where a few of many experts' matrices are read
        _part("experts_prompt", "experts", 2048),
        _part("experts_decode", "experts", 1, requests=8),
        # latent attention: a whole prompt, and a decode step of 16 requests
        _part("latent_prompt", "latent", 2048),
        _part("latent_decode", "latent", 1, past=1500, requests=16),
        # the recurrences over prompts: one long, several ragged, one of odd length
        _part("mlstm_prompt", "mlstm", 2048),
        _part("mamba2_prompts", "mamba2", 777, requests=3),
        _part("channel_delta_prompt", "channel_delta", 1531),
        # differential attention over a portion that follows cached tokens (the window crosses the border)
        _part("diff_attention_portion", "diff_attention", 1500, past=500),
    ]


def _between(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["prompt", "replies"] + 2 * sorted(PARTS))
    if what == "prompt":
        return {"kind": "prompt", "model": "1b", "dtype": "bfloat16", "tokens": _between(rng, 16, 2048)}
    if what == "replies":
        model = rng.choice(["1b", "tiny"])
        return {"kind": "replies", "model": model, "dtype": "float32" if model == "tiny" else "bfloat16", "requests": rng.randint(1, 8),
                "prompt": _between(rng, 2, 100 if model == "tiny" else 200), "steps": rng.randint(2, 8)}
    size = rng.choice(["large", "large", "small"])
    dtype = "float32" if what not in ("experts",) and rng.random() < 0.1 else "bfloat16"
    if rng.random() < 0.35:        # a decode step
        case = _part("", what, 1, past=0 if what == "experts" else _between(rng, 32, 2000 if what not in STATEFUL else 100),
                     requests=_between(rng, 1, 64 if what != "latent" else 32), size=size, dtype=dtype)
    else:                          # portions of prompts
        requests = rng.choice([1, 1, 2, 4])
        new = _between(rng, 16, (2048 if dtype == "bfloat16" else 256) // requests)
        case = _part("", what, new, past=rng.choice([0, 0, _between(rng, 16, 1000)]) if what != "experts" else 0, requests=requests, size=size,
                     dtype=dtype)
    del case["name"]
    return case


# ------------------------------------------------------------------ named tensors
def _tensor(seed, name, shape, std=1.0, mean=0.0, dtype=BF16):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (2 ** 62))
    return (torch.randn(shape, generator=g, device="cuda", dtype=F32) * std + mean).to(dtype)


def _uniform(seed, name, shape, lo, hi):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (2 ** 62))
    return torch.rand(shape, generator=g, device="cuda", dtype=F32) * (hi - lo) + lo


def _matrix(seed, name, rows, cols, gain=1.0):
    return _tensor(seed, name, (rows, cols), gain * cols ** -0.5)


def _step_bias(seed, name, shape):
    """What softplus turns into step sizes of 0.001 to 0.1, evenly over their logarithm."""
    dt = torch.exp(_uniform(seed, name, shape, math.log(1e-3), math.log(1e-1)))
    return torch.log(torch.expm1(dt)).to(BF16)


def _llama_tensors(m, seed):
    d, f, hd = m["hidden_size"], m["intermediate_size"], m["head_dim"]
    H, G = m["num_attention_heads"], m["num_key_value_heads"]
    t = {"model.embed_tokens.weight": _tensor(seed, "embed", (m["vocab_size"], d)), "model.norm.weight": _tensor(seed, "norm", (d,), 0.1, 1.0)}
    for i in range(m["num_hidden_layers"]):
        p = "model.layers.%d." % i
        t[p + "input_layernorm.weight"] = _tensor(seed, p + "n1", (d,), 0.1, 1.0)
        t[p + "post_attention_layernorm.weight"] = _tensor(seed, p + "n2", (d,), 0.1, 1.0)
        for n, rows, cols in (("self_attn.q_proj", H * hd, d), ("self_attn.k_proj", G * hd, d), ("self_attn.v_proj", G * hd, d),
                              ("self_attn.o_proj", d, H * hd), ("mlp.gate_proj", f, d), ("mlp.up_proj", f, d), ("mlp.down_proj", d, f)):
            t[p + n + ".weight"] = _matrix(seed, p + n, rows, cols)
    if not m["tie_word_embeddings"]:
        t["lm_head.weight"] = _matrix(seed, "head", m["vocab_size"], d)
    return t


def _mixer_tensors(part, s, seed):
    """The tensors of one mixer or feed-forward by their short names."""
    w = s["width"]
    M = lambda n, r, c, gain=1.0: (n, _matrix(seed, n, r, c, gain))
    V = lambda n, k, std, mean=0.0: (n, _tensor(seed, n, (k,), std, mean))
    if part == "experts":
        t = [M("router", s["experts"], w), M("shared.gate", s["shared"], w), M("shared.up", s["shared"], w), M("shared.down", w, s["shared"]),
             M("shared.sg", 1, w)]
        for e in range(s["experts"]):
            t += [M("e%d.gate" % e, s["ff"], w), M("e%d.up" % e, s["ff"], w), M("e%d.down" % e, w, s["ff"])]
        return dict(t)
    if part == "latent":
        H = s["heads"]
        return dict([M("q", H * (s["dim"] + s["rot"]), w), M("dkv", s["rank"] + s["rot"], w), V("dkv.norm", s["rank"], 0.1, 1.0),
                     M("uk", H * s["dim"], s["rank"]), M("uv", H * s["vdim"], s["rank"]), M("g", H * s["vdim"], w), M("o", w, H * s["vdim"])])
    if part == "mlstm":
        H, n, dv = s["heads"], s["dim"], s["vdim"]
        return dict([M("q", H * n, w), M("k", H * n, w), M("v", H * dv, w), M("g", H * dv, w), M("o", w, H * dv), V("norm", H * dv, 0.1, 1.0),
                     M("i", H, w), V("i.b", H, 1.0), M("f", H, w), V("f.b", H, 1.0, 3.0)])
    if part == "mamba2":
        H, inner = s["heads"], s["heads"] * s["vdim"]
        ch = inner + 2 * s["state"]
        return dict([M("in", inner + ch + H, w), ("conv", _tensor(seed, "conv", (ch, s["taps"]), 0.5)), V("conv.b", ch, 0.1),
                     ("dt_bias", _step_bias(seed, "dt_bias", (H,))), ("A_log", torch.log(_uniform(seed, "A_log", (H,), 1, 16)).to(BF16)),
                     V("D", H, 0.1, 1.0), V("norm", inner, 0.1, 1.0), M("o", w, inner)])
    if part == "channel_delta":
        H, G, n, r = s["heads"], s["kv"], s["dim"], s["rank"]
        t = [M("q", G * n, w), M("k", G * n, w), M("v", H * n, w), M("b", H, w), M("a1", r, w), M("a2", H * n, r, 0.5), M("g1", r, w),
             M("g2", H * n, r), V("norm", n, 0.1, 1.0), M("o", w, H * n), ("dt_bias", _step_bias(seed, "dt_bias", (H * n,))),
             ("A_log", torch.log(_uniform(seed, "A_log", (H,), 1, 16)).to(BF16))]
        return dict(t + [(x + ".conv", _tensor(seed, x + ".conv", (c, s["taps"]), 0.5)) for x, c in (("q", G * n), ("k", G * n), ("v", H * n))])
    H, G, n, dv = s["heads"], s["kv"], s["dim"], s["vdim"]
    t = [M("q", H * 2 * n, w), M("k", G * 2 * n, w), M("v", G * dv, w), M("o", w, H * dv), V("q.norm", n, 0.1, 1.0), V("k.norm", n, 0.1, 1.0)]
    t += [V(x + ".b", c, 0.1) for x, c in (("q", H * 2 * n), ("k", G * 2 * n), ("v", G * dv))]
    return dict(t + [V(x, n, 0.1) for x in ("lq1", "lk1", "lq2", "lk2")])


def _part_model(part, s, seed, dtype):
    """(configuration, tensors) of a one-layer model around the part."""
    w, vocab = s["width"], 512
    if part == "attention":
        raw = dict(MODELS["1b"], vocab_size=vocab, hidden_size=w, intermediate_size=256, num_hidden_layers=1, num_attention_heads=s["heads"],
                   num_key_value_heads=s["kv"], head_dim=s["dim"])
        return raw, _llama_tensors(raw, seed)
    short = _mixer_tensors(part, s, seed)
    p = "l0.mlp." if part == "experts" else "l0.mix."
    t = {p + k: v for k, v in short.items()}
    t.update({"embed": _tensor(seed, "embed", (vocab, w)), "final.norm": torch.ones(w, device="cuda", dtype=BF16)})
    raw = {"vocab": vocab, "width": w, "norm": {"eps": EPS}}
    if part == "channel_delta":
        mixer = dict(heads=s["heads"], kv_heads=s["kv"], dim=s["dim"], vdim=s["dim"], conv=s["taps"], decay_rank=s["rank"], gate_rank=s["rank"])
        raw.update(architecture="Lugizen", canon={"taps": s["taps"]}, layers=[{"type": part, "mixer": mixer, "mlp": None}])
        t["l0.canon1"] = _tensor(seed, "canon1", (w, s["taps"]), 0.3)
        t["l0.norm1"], t["final.norm"] = torch.ones((), device="cuda", dtype=BF16), torch.ones((), device="cuda", dtype=BF16)
        t["head"] = _matrix(seed, "head", vocab, w)
    elif part == "diff_attention":
        mixer = dict(heads=s["heads"], kv_heads=s["kv"], dim=s["dim"], vdim=s["vdim"], scale=0.125, diff=0.2, mask={"size": s["window"]}, rot=ROT)
        raw.update(architecture="Lotirax", layers=[{"type": "attention", "mixer": mixer, "mlp": None}])
        t["final.norm"] = torch.zeros(w, device="cuda", dtype=BF16)
        t["l0.norm1"], t["l0.ls1"] = torch.zeros(w, device="cuda", dtype=BF16), torch.ones(w, device="cuda", dtype=BF16)
    else:
        kind, mlp = part, None
        if part == "latent":
            kind, mixer = "latent_attention", dict(heads=s["heads"], dim=s["dim"], rot_dim=s["rot"], vdim=s["vdim"], kv_rank=s["rank"],
                                                   scale=(s["dim"] + s["rot"]) ** -0.5, rot={"base": 10000.0, "dims": s["rot"]})
        elif part == "mamba2":
            mixer = dict(heads=s["heads"], vdim=s["vdim"], state=s["state"], groups=1, conv=s["taps"], norm_groups=1)
        else:                      # the experts stand beside a small recurrence
            small = dict(width=w, heads=1, dim=16, vdim=16)
            m = s if part == "mlstm" else small
            kind, mixer = "mlstm", dict(heads=m["heads"], dim=m["dim"], vdim=m["vdim"], gate_cap=15.0)
            if part == "experts":
                t.update({"l0.mix." + k: v for k, v in _mixer_tensors("mlstm", small, seed).items()})
                t["l0.norm2"] = torch.ones(w, device="cuda", dtype=BF16)
                mlp = {"kind": "moe", "expert": {"ff": s["ff"]}, "router": {"experts": s["experts"], "top": s["top"]}, "shared": {"ff": s["shared"]}}
        raw.update(architecture="Deganex", layers=[{"type": kind, "mixer": mixer, "mlp": mlp}])
        t["l0.norm1"], t["head"] = torch.ones(w, device="cuda", dtype=BF16), _matrix(seed, "head", vocab, w)
    if dtype == F32:
        t = {k: v.float() for k, v in t.items()}
    return raw, t


def _runner(raw, tensors, dtype, max_tokens, requests, max_len):
    name = raw.get("architecture") or raw["architectures"][0]
    config = lookup_architecture(name).config_from_dict(raw)
    return ModelRunner(config=config, tensors=tensors, dtype=dtype, max_tokens=max_tokens, max_requests=requests, max_model_len=max_len)


# ------------------------------------------------------------------ what a pass brings
def _lengths(case):
    """(cached tokens, new tokens) of each request: the first as the case says, later ones down to half."""
    R = case["requests"]
    cut = lambda n, i: n - (i * n) // (2 * R)
    return [(cut(case["past"], i), max(1, cut(case["new"], i))) for i in range(R)]


def _inputs(case, seed):
    """Each request's layer inputs [past + new, width], as a norm (or, ahead of an input convolution, the stream) leaves them."""
    s = PARTS[case["part"]][case["size"]]
    dtype = F32 if case["part"] == "channel_delta" else DTYPES[case["dtype"]]
    return [_tensor(seed, "x%d" % i, (p + n, s["width"]), dtype=BF16).to(dtype) for i, (p, n) in enumerate(_lengths(case))]


def _ids(case, seed):
    """Prompts and the tokens of the steps that follow, per request."""
    m = MODELS[case["model"]]
    if case["kind"] == "prompt":
        want = [case["tokens"]]
    else:
        want = [max(1, case["prompt"] - (3 * i) % max(1, case["prompt"])) + case["steps"] for i in range(case["requests"])]
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, m["vocab_size"], (n,), generator=g).tolist() for n in want]


def prepare(case, seed):
    if case["kind"] != "part":
        m = MODELS[case["model"]]
        ids = _ids(case, seed)
        total = sum(len(x) + 16 for x in ids)
        tensors = _llama_tensors(m, seed)
        if case["dtype"] == "float32":
            tensors = {k: v.float() for k, v in tensors.items()}
        state = {"case": case, "ids": ids, "runner": _runner(m, tensors, case["dtype"], total, len(ids), max(len(x) for x in ids))}
        if case["kind"] == "replies":
            run(state)             # an engine at work has captured its decode step
        return state

    part, s, dtype = case["part"], PARTS[case["part"]][case["size"]], DTYPES[case["dtype"]]
    raw, tensors = _part_model(part, s, seed, dtype)
    lengths = _lengths(case)
    longest = max(p + n for p, n in lengths)
    captured = case["new"] == 1
    r = _runner(raw, tensors, case["dtype"], sum(-(-(p + n) // 16) * 16 for p, n in lengths), len(lengths), longest)
    del tensors
    block = r.model.blocks[0]
    layer = block.feed_forward if part == "experts" else block.mixer
    more = (2, 3) if part == "channel_delta" else ()           # its convolutions' tails (1 would be the embedding's own state: none)
    views = [r.cache.layer_view(i) for i in (0,) + more]
    view = views[0] if len(views) == 1 else CompositeCacheView(views=views)
    call = (lambda x, ctx: layer.forward(x, ctx)) if part == "experts" else (lambda x, ctx: layer.forward(x, ctx, view))
    xs = _inputs(case, seed)
    for i, (p, _) in enumerate(lengths):                       # what earlier steps left in the cache
        if p and part != "experts":
            ctx = r.prepare([StepEntry(i, [0] * p)])
            call(xs[i][:p].contiguous(), ctx)
            r.cache.commit(i, p)
    ctx = r.prepare([StepEntry(i, [0] * n) for i, (_, n) in enumerate(lengths)])
    x = torch.cat([xs[i][p:] for i, (p, _) in enumerate(lengths)]).contiguous()
    states = [v.tensor for v in views] if part in STATEFUL else []
    state = {"case": case, "runner": r, "ctx": ctx, "x": x, "call": call, "states": states, "before": [t.clone() for t in states]}
    if captured:
        ctx.captured = True
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _pass(state)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["out"] = _pass(state)
    return state


def _pass(state):
    for t, b in zip(state["states"], state["before"]):         # the requests' states as their earlier tokens left them
        t.copy_(b)
    y = state["call"](state["x"], state["ctx"])
    return [y] + state["states"]


def run(state):
    case = state["case"]
    if case["kind"] == "part":
        if "graph" in state:
            state["graph"].replay()
            return state["out"]
        return _pass(state)
    r, ids = state["runner"], state["ids"]
    if case["kind"] == "prompt":
        return [r.step([StepEntry(0, ids[0], [len(ids[0]) - 1])], end=[0])]
    n = case["steps"]
    who = range(len(ids))
    out = [r.step([StepEntry(i, ids[i][:-n], [len(ids[i]) - n - 1]) for i in who])]
    for k in range(n):
        out.append(r.step([StepEntry(i, [ids[i][len(ids[i]) - n + k]], [0]) for i in who], end=who if k == n - 1 else ()))
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _pairs(case, window=0):
    seen = lambda pos: min(pos + 1, window) if window else pos + 1
    return sum(seen(p + j) for p, n in _lengths(case) for j in range(n))


def work(case):
    if case["kind"] != "part":
        m = MODELS[case["model"]]
        d, f, hd, L = m["hidden_size"], m["intermediate_size"], m["head_dim"], m["num_hidden_layers"]
        H, G, V = m["num_attention_heads"], m["num_key_value_heads"], m["vocab_size"]
        e = 4 if case["dtype"] == "float32" else 2
        layer, head = 2 * d * H * hd + 2 * d * G * hd + 3 * d * f, V * d
        lens = [len(x) for x in _ids(case, 0)]
        n = case.get("steps", 0)
        kv = lambda total: total * L * 2 * G * hd * e
        nbytes = (L * layer + head) * e * (1 + n) + len(lens) * V * 4 * (1 + n) + kv(sum(lens))
        flops = 2.0 * sum(lens) * L * layer + 2.0 * len(lens) * (1 + n) * head + sum(4.0 * L * H * hd * x * (x + 1) / 2 for x in lens)
        for k in range(n):
            nbytes += kv(sum(x - n + k for x in lens))
        return {"bytes": nbytes, "flops": flops}
    part, s = case["part"], PARTS[case["part"]][case["size"]]
    e = 4 if case["dtype"] == "float32" else 2
    w, T, R = s["width"], sum(n for _, n in _lengths(case)), case["requests"]
    rows = sum(p + n for p, n in _lengths(case))
    io = 2 * T * w * e
    if part == "attention":
        weights, kv = w * s["dim"] * 2 * (s["heads"] + s["kv"]), 2 * s["kv"] * s["dim"]
        return {"bytes": io + (weights + rows * kv) * e, "flops": 2.0 * T * weights + 4.0 * s["heads"] * s["dim"] * _pairs(case)}
    if part == "experts":
        one, shared = 3 * w * s["ff"], 3 * w * s["shared"]
        touched = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** T)
        return {"bytes": T * w * (e + 4) + (touched * one + shared + s["experts"] * w) * e,
                "flops": 2.0 * T * (s["top"] * one + shared + s["experts"] * w)}
    if part == "latent":
        H, n, rd, dv, rank = s["heads"], s["dim"], s["rot"], s["vdim"], s["rank"]
        dense = w * (H * (n + rd) + rank + rd + 2 * H * dv)
        up = H * (n + dv) * rank
        pairs = _pairs(case)
        expanded = 2.0 * rows * up + 2.0 * H * pairs * (n + rd + dv)               # keys and values formed from the latents once
        carried = 2.0 * T * up + 2.0 * H * pairs * (2 * rank + rd)                 # or the queries carried into the latent space
        return {"bytes": io + (dense + up + rows * (rank + rd)) * e, "flops": 2.0 * T * dense + min(expanded, carried)}
    if part == "diff_attention":
        H, G, n, dv = s["heads"], s["kv"], s["dim"], s["vdim"]
        weights, row = w * (2 * n * (H + G) + G * dv + H * dv), G * (2 * n + dv)
        read = sum(min(p + m, s["window"] + m - 1) for p, m in _lengths(case))
        return {"bytes": io + (weights + read * row) * e, "flops": 2.0 * T * weights + H * _pairs(case, s["window"]) * (4.0 * n + 4.0 * dv)}
    if part == "mlstm":
        H, n, dv = s["heads"], s["dim"], s["vdim"]
        weights, st = w * (2 * H * n + 3 * H * dv + 2 * H), H * n * dv
    elif part == "mamba2":
        H, inner = s["heads"], s["heads"] * s["vdim"]
        weights, st = w * (3 * inner + 2 * s["state"] + H), inner * s["state"]
    else:
        H, G, n, r = s["heads"], s["kv"], s["dim"], s["rank"]
        weights, st = w * (2 * G * n + 2 * H * n + H + 2 * r) + 2 * r * H * n, H * n * n
        io = T * w * (4 + e)
    per = 6.0 if part == "channel_delta" else 4.0              # the delta rule also reads the state at every key
    return {"bytes": io + weights * e + 2 * R * st * 4, "flops": 2.0 * T * weights + per * T * st}


def tolerance(case):
    # 32-bit sums; the matrices' products and the exponentials' arguments add up over a layer, the tiny model has three of them
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-3}
    # a whole model in bfloat16: what one layer rounds otherwise travels through the fifteen behind it
    if case["kind"] != "part":
        return {"rel": 3e-2, "max": 3e-1}
    return {"rel": 1e-2, "max": 4e-1}


# ------------------------------------------------------------------ the same in 64 bits
def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _softmax_rows(s, lo, window=0):
    """Softmax of scores [.., n, keys]: query row i stands at key lo + i."""
    i = torch.arange(s.shape[-2], device="cuda")[:, None] + lo
    j = torch.arange(s.shape[-1], device="cuda")[None, :]
    hide = (j > i) | ((i - j >= window) if window else torch.zeros_like(j, dtype=torch.bool))
    return torch.softmax(s.masked_fill(hide, -math.inf), dim=-1)


def _turn(x, pos, freq, pairs, mag=1.0):
    """Rotates pairs of entries of the last axis of x [T, heads, n]; pairs: 'halves' (i, i + dims/2) or 'neighbours' (2i, 2i + 1)."""
    a = pos[:, None].to(F64) * freq[None, :]
    c, s = (torch.cos(a) * mag)[:, None, :], (torch.sin(a) * mag)[:, None, :]
    k = freq.numel()
    out = x.clone()
    u, v = (x[..., :k], x[..., k: 2 * k]) if pairs == "halves" else (x[..., 0: 2 * k: 2], x[..., 1: 2 * k: 2])
    if pairs == "halves":
        out[..., :k], out[..., k: 2 * k] = u * c - v * s, v * c + u * s
    else:
        out[..., 0: 2 * k: 2], out[..., 1: 2 * k: 2] = u * c - v * s, v * c + u * s
    return out


def _frequencies(dims, base):
    return torch.tensor([float(base) ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64, device="cuda")


def _llama_frequencies(m):
    sc, out = m["rope_scaling"], []
    for i in range(m["head_dim"] // 2):
        f = m["rope_theta"] ** (-2.0 * i / m["head_dim"])
        turns = sc["original_max_position_embeddings"] * f / (2 * math.pi)          # over the original length
        mix = min(1.0, max(0.0, (turns - sc["low_freq_factor"]) / (sc["high_freq_factor"] - sc["low_freq_factor"])))
        out.append((1 - mix) * f / sc["factor"] + mix * f)
    return torch.tensor(out, dtype=F64, device="cuda")


def _yarn_frequencies(rot):
    dims, base, sc, out = rot["dims"], rot["base"], rot["scaling"], []
    turn = lambda t: dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(base))
    lo, hi = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), dims - 1)
    for i in range(dims // 2):
        f, ramp = base ** (-2.0 * i / dims), min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        out.append(f / sc["factor"] * ramp + f * (1 - ramp))
    return torch.tensor(out, dtype=F64, device="cuda"), 0.1 * math.log(sc["factor"]) + 1.0


def _grouped_attention(q, k, v, scale, lo, window=0):
    """q [n, H, d], k [keys, G, d], v [keys, G, m] -> [n, H * m]; the first query stands at key lo."""
    H, G = q.shape[1], k.shape[1]
    out = [_softmax_rows(q[:, h] @ k[:, h // (H // G)].T * scale, lo, window) @ v[:, h // (H // G)] for h in range(H)]
    return torch.cat(out, dim=1)


def _llama_attention(h, W, p, m, lo=0):
    T, hd = h.shape[0], m["head_dim"]
    H, G = m["num_attention_heads"], m["num_key_value_heads"]
    w = lambda n: W[p + "self_attn." + n + "_proj.weight"].to(F64)
    pos, freq = torch.arange(T, device="cuda"), _llama_frequencies(m)
    q = _turn((h[lo:] @ w("q").T).reshape(T - lo, H, hd), pos[lo:], freq, "halves")
    k = _turn((h @ w("k").T).reshape(T, G, hd), pos, freq, "halves")
    v = (h @ w("v").T).reshape(T, G, hd)
    return _grouped_attention(q, k, v, hd ** -0.5, lo) @ w("o").T


def _llama_stream(m, W, ids):
    eps = m["rms_norm_eps"]
    x = W["model.embed_tokens.weight"][torch.tensor(ids, device="cuda")].to(F64)
    for i in range(m["num_hidden_layers"]):
        p = "model.layers.%d." % i
        x = x + _llama_attention(_unit(x, eps) * W[p + "input_layernorm.weight"].to(F64), W, p, m)
        h = _unit(x, eps) * W[p + "post_attention_layernorm.weight"].to(F64)
        w = lambda n: W[p + "mlp." + n + "_proj.weight"].to(F64)
        x = x + (_silu(h @ w("gate").T) * (h @ w("up").T)) @ w("down").T
    return _unit(x, eps) * W["model.norm.weight"].to(F64)


def _experts(h, W, s):
    logits = h @ W["router"].T
    top = torch.topk(logits, s["top"], dim=1)
    weight = torch.softmax(top.values, dim=1)
    out = torch.sigmoid(h @ W["shared.sg"].T) * ((_silu(h @ W["shared.gate"].T) * (h @ W["shared.up"].T)) @ W["shared.down"].T)
    for e in range(s["experts"]):
        at, slot = (top.indices == e).nonzero(as_tuple=True)
        x = h[at]
        y = (_silu(x @ W["e%d.gate" % e].to(F64).T) * (x @ W["e%d.up" % e].to(F64).T)) @ W["e%d.down" % e].to(F64).T
        out.index_add_(0, at, weight[at, slot][:, None] * y)
    return out


def _latent(h, W, s, lo):
    T, H, n, rd, dv, rank = h.shape[0], s["heads"], s["dim"], s["rot"], s["vdim"], s["rank"]
    pos, freq = torch.arange(T, device="cuda"), _frequencies(rd, 10000.0)
    q = (h[lo:] @ W["q"].T).reshape(T - lo, H, n + rd)
    q = torch.cat([q[..., :n], _turn(q[..., n:], pos[lo:], freq, "neighbours")], dim=-1)
    down = h @ W["dkv"].T
    c = _unit(down[:, :rank], EPS) * W["dkv.norm"]
    kr = _turn(down[:, None, rank:], pos, freq, "neighbours")
    k = torch.cat([(c @ W["uk"].T).reshape(T, H, n), kr.expand(T, H, rd)], dim=-1)
    y = _grouped_attention(q, k, (c @ W["uv"].T).reshape(T, H, dv), (n + rd) ** -0.5, lo)
    return (y * torch.sigmoid(h[lo:] @ W["g"].T)) @ W["o"].T


def _mlstm(h, W, s, lo):
    T, H, n, dv, cap = h.shape[0], s["heads"], s["dim"], s["vdim"], 15.0
    q, k, v = (h @ W["q"].T).reshape(T, H, n) * n ** -0.5, (h @ W["k"].T).reshape(T, H, n), (h @ W["v"].T).reshape(T, H, dv)
    li = cap * torch.tanh((h @ W["i"].T + W["i.b"]) / cap)
    lf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ W["f"].T + W["f.b"]) / cap))
    # the running maximum m_t = max(lf_t + m_(t-1), li_t), m_(-1) = 0, from prefix sums of the forget gates
    F = torch.cumsum(lf, 0)
    m = F + torch.clamp(torch.cummax(li - F, 0).values, min=0.0)
    before = torch.cat([torch.zeros(1, H, dtype=F64, device="cuda"), m[:-1]])
    keep, take = torch.exp(lf + before - m), torch.exp(li - m)
    S, N, out = torch.zeros(H, n, dv, dtype=F64, device="cuda"), torch.zeros(H, n, dtype=F64, device="cuda"), []
    for t in range(T):
        S = keep[t][:, None, None] * S + (take[t][:, None] * k[t])[:, :, None] * v[t][:, None, :]
        N = keep[t][:, None] * N + take[t][:, None] * k[t]
        if t >= lo:
            out.append((q[t][:, None, :] @ S)[:, 0] / (torch.maximum((N * q[t]).sum(-1).abs(), torch.exp(-m[t])) + 1e-6)[:, None])
    y = _unit(torch.stack(out), EPS).reshape(T - lo, H * dv) * W["norm"] * torch.sigmoid(h[lo:] @ W["g"].T)
    return y @ W["o"].T


def _conv(x, w):
    taps = w.shape[1]
    xx = torch.cat([torch.zeros(taps - 1, x.shape[1], dtype=F64, device="cuda"), x])
    return sum(xx[j: j + x.shape[0]] * w[:, j] for j in range(taps))


def _mamba2(h, W, s, lo):
    T, H, P, N = h.shape[0], s["heads"], s["vdim"], s["state"]
    inner = H * P
    proj = h @ W["in"].T
    z, xbc, dt = proj[:, :inner], proj[:, inner: 2 * inner + 2 * N], proj[:, 2 * inner + 2 * N:]
    conv = _silu(_conv(xbc, W["conv"]) + W["conv.b"])
    x, B, C = conv[:, :inner].reshape(T, H, P), conv[:, inner: inner + N], conv[:, inner + N:]
    step = torch.nn.functional.softplus(dt + W["dt_bias"])
    keep = torch.exp(-torch.exp(W["A_log"]) * step)
    S, out = torch.zeros(H, N, P, dtype=F64, device="cuda"), []
    for t in range(T):
        S = keep[t][:, None, None] * S + B[t][None, :, None] * (step[t][:, None] * x[t])[:, None, :]
        if t >= lo:
            out.append(C[t] @ S)
    y = (torch.stack(out) + W["D"][:, None] * x[lo:]).reshape(T - lo, inner) * _silu(z[lo:])
    return (_unit(y, EPS) * W["norm"]) @ W["o"].T


def _channel_delta(x, W, canon, s, lo):
    h = x + _conv(x, canon)
    T, H, G, n = h.shape[0], s["heads"], s["kv"], s["dim"]
    q, k, v = (_silu(_conv(h @ W[c].T, W[c + ".conv"])).reshape(T, heads, n) for c, heads in (("q", G), ("k", G), ("v", H)))
    length = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + KEY_EPS)
    q, k = ((length(t)).repeat_interleave(H // G, dim=1) for t in (q, k))
    q = q * n ** -0.5
    beta = torch.sigmoid(h @ W["b"].T)
    z = (h @ W["a1"].T) @ W["a2"].T + W["dt_bias"]
    decay = torch.exp(-torch.exp(W["A_log"]).repeat_interleave(n) * torch.nn.functional.softplus(z)).reshape(T, H, n)
    S, out = torch.zeros(H, n, n, dtype=F64, device="cuda"), []
    for t in range(T):
        S = decay[t][:, :, None] * S
        u = beta[t][:, None] * (v[t] - (k[t][:, None, :] @ S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None, :]
        if t >= lo:
            out.append((q[t][:, None, :] @ S)[:, 0])
    y = _unit(torch.stack(out), EPS) * W["norm"] * torch.sigmoid((h[lo:] @ W["g1"].T) @ W["g2"].T).reshape(T - lo, H, n)
    return y.reshape(T - lo, H * n) @ W["o"].T


def _diff(h, W, s, lo):
    T, H, G, n, dv = h.shape[0], s["heads"], s["kv"], s["dim"], s["vdim"]
    pos = torch.arange(T, device="cuda")
    freq, mag = _yarn_frequencies(ROT)
    turned = lambda c, heads, rows: _turn((_unit((h[rows:] @ W[c].T + W[c + ".b"]).reshape(-1, heads, n), EPS) * W[c + ".norm"]), pos[rows:],
                                          freq, "halves", mag).reshape(-1, heads // 2, 2, n)
    q, k, v = turned("q", 2 * H, lo), turned("k", 2 * G, 0), (h @ W["v"].T + W["v.b"]).reshape(T, G, dv)
    lam = math.exp(float((W["lq1"] * W["lk1"]).sum())) - math.exp(float((W["lq2"] * W["lk2"]).sum())) + 0.2
    a1, a2 = (_grouped_attention(q[:, :, i], k[:, :, i], v, 0.125, lo, s["window"]) for i in (0, 1))
    return (_unit((a1 - lam * a2).reshape(-1, H, dv), EPS) * 0.8).reshape(-1, H * dv) @ W["o"].T


def exact(case, seed):
    if case["kind"] != "part":
        m, ids = MODELS[case["model"]], _ids(case, seed)
        W = _llama_tensors(m, seed)
        n = case.get("steps", 0)
        rows = [_llama_stream(m, W, x)[len(x) - n - 1:] for x in ids]                # [1 + steps, width] of each request
        head = W["model.embed_tokens.weight"].to(F64)
        return [torch.stack([r[k] for r in rows]) @ head.T for k in range(1 + n)]
    part, s = case["part"], PARTS[case["part"]][case["size"]]
    xs, lengths = _inputs(case, seed), _lengths(case)
    if part == "attention":
        raw, W = _part_model(part, s, seed, BF16)
        return [torch.cat([_llama_attention(x.to(F64), W, "model.layers.0.", raw, p) for x, (p, _) in zip(xs, lengths)])]
    W = _mixer_tensors(part, s, seed)
    W = W if part == "experts" else {k: v.to(F64) for k, v in W.items()}
    if part == "experts":
        W = {k: v if k[0] == "e" else v.to(F64) for k, v in W.items()}
        return [_experts(torch.cat([x[p:] for x, (p, _) in zip(xs, lengths)]).to(F64), W, s)]
    if part == "channel_delta":
        canon = _tensor(seed, "canon1", (s["width"], s["taps"]), 0.3).to(F64)
        f = lambda x, p: _channel_delta(x, W, canon, s, p)
    else:
        g = {"latent": _latent, "mlstm": _mlstm, "mamba2": _mamba2, "diff_attention": _diff}[part]
        f = lambda x, p: g(x, W, s, p)
    y = torch.cat([f(x.to(F64), p) for x, (p, _) in zip(xs, lengths)])
    return [y] + [None] * {"mlstm": 1, "mamba2": 1, "channel_delta": 3}.get(part, 0)
