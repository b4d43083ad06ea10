"""Timed cases of the engine: what a program that serves models with it has it do, step by step.

Every case is one pass through ``StepEngine.step`` (and ``DeviceSampler`` where tokens are drawn on the device) over a
model with random weights at the layer sizes of this repository's benchmark. ``exact`` computes the same logits in
64 bits with plain torch, whole sequences at once, from the same weights and tokens.
"""
import math
import re
import zlib

import torch

VOCAB = 128256
PAGE = 16
STEP_TOKENS = 2048           # rows of a step while a context is filled, and of a portion of a long prompt

# The layer sizes of the benchmark's three shapes.
SIZES = {
    "1b": {"width": 2048, "ff": 8192, "heads": 32, "kv_heads": 8, "head_dim": 64, "tied": True, "factor": 32.0},
    "3b": {"width": 3072, "ff": 8192, "heads": 24, "kv_heads": 8, "head_dim": 128, "tied": True, "factor": 32.0},
    "8b": {"width": 4096, "ff": 14336, "heads": 32, "kv_heads": 8, "head_dim": 128, "tied": False, "factor": 8.0},
}
DESIGNS = ("nipadra", "gekupel", "pinorax", "fovezen", "mimolix", "kidarax")
ROUTED = ("gekupel", "mimolix", "kidarax")        # their routers read the stream (Pinorax looks its experts up)


# ---------------------------------------------------------------------------------------------------- the cases
def listed():
    llama = {"arch": "llama", "size": "1b", "layers": 16, "dtype": "bfloat16", "tokens": 0, "new": 1, "ragged": False}
    design = {"size": "1b", "layers": 4, "dtype": "bfloat16", "mode": "requests", "tokens": 0, "ragged": True}
    return [
        # one user in a chat, early in the text: the latency of a token, all launches and weights
        dict(llama, name="decode_b1_short", mode="decode", requests=1, context=130),
        # the serving load of the benchmark: eight long contexts, a token each
        dict(llama, name="decode_b8_long", mode="decode", requests=8, context=8191),
        # a full batch of requests at different places of their texts
        dict(llama, name="decode_b64_ragged", mode="decode", requests=64, context=1900, ragged=True),
        # an ordinary prompt in one step, up to its first token
        dict(llama, name="prefill_2048", mode="prefill", requests=1, context=0, tokens=2048),
        # a long document into a model with heads of 128, in portions
        dict(llama, name="prefill_long_8b", size="8b", layers=8, mode="prefill", requests=1, context=0, tokens=6001),
        # continuous batching: a portion of someone's prompt beside everyone else's next token
        dict(llama, name="mixed_3b", size="3b", layers=14, mode="mixed", requests=23, context=1500, tokens=489, ragged=True),
        # the true 32-bit path: short prompts, then tokens drawn on the device and fed back from there
        dict(llama, name="float32_sampled", layers=4, dtype="float32", mode="sampled", requests=6, context=90, new=5, ragged=True),
        # the other designs, each as requests come: prompts of several users in one step, then a token each for some steps.
        # linear attention and state space beside a window
        dict(design, name="nipadra_requests", arch="nipadra", requests=3, context=900, new=8),
        # latent attention, blocks with a distance bias, routed experts
        dict(design, name="gekupel_requests", arch="gekupel", requests=8, context=301, new=8),
        # copies of the stream, decays per row, capped scores over a window
        dict(design, name="fovezen_requests", arch="fovezen", requests=1, context=2048, new=8, ragged=False),
        # the gated delta rule, two score maps
        dict(design, name="mimolix_requests", arch="mimolix", requests=4, context=512, new=8),
        # retention, gated and latent attention, experts whose weights scale their inputs
        dict(design, name="kidarax_requests", arch="kidarax", requests=2, context=1300, new=8),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.5:
        size = rng.choice(("1b", "1b", "3b", "8b"))
        case = {"arch": "llama", "size": size, "layers": rng.randint(2, {"1b": 16, "3b": 12, "8b": 8}[size]), "dtype": "bfloat16",
                "tokens": 0, "new": 1, "ragged": rng.random() < 0.7}
        mode = rng.choice(("decode", "decode", "prefill", "mixed"))
        if mode == "prefill":
            return dict(case, mode=mode, requests=1, context=0, tokens=_log(rng, 17, 6001))
        requests = _log(rng, 1, 64)
        case.update(mode=mode, requests=requests, context=_log(rng, 16, min(8191, 65528 // requests)))
        if mode == "mixed":
            case["tokens"] = _log(rng, 17, STEP_TOKENS - requests)
        return case
    if pick < 0.6:
        return {"arch": "llama", "size": "1b", "layers": rng.randint(2, 6), "dtype": "float32", "mode": "sampled", "tokens": 0,
                "requests": _log(rng, 1, 8), "context": _log(rng, 8, 128), "new": rng.randint(2, 6), "ragged": rng.random() < 0.7}
    requests = _log(rng, 1, 16)
    return {"arch": rng.choice(DESIGNS), "size": rng.choice(("1b", "1b", "8b")), "layers": 4, "dtype": "bfloat16", "mode": "requests",
            "tokens": 0, "requests": requests, "context": _log(rng, 16, STEP_TOKENS // requests), "new": rng.randint(2, 8),
            "ragged": rng.random() < 0.7}


def _lengths(case):
    """Cached positions (decode, mixed) or prompt lengths (requests, sampled) of the case's requests."""
    n, c = case["requests"], case["context"]
    if not case["ragged"] or n == 1:
        return [c] * n
    return [max(1, int(c * (0.2 + 0.8 * ((i * 0.6180339887) % 1.0)))) for i in range(n)]


# ---------------------------------------------------------------------------------------------------- configurations
def config_of(case):
    """config.json of the case's model: the benchmark's shape of that design."""
    s, n, arch = SIZES[case["size"]], case["layers"], case["arch"]
    D, ff, H, G, hd = s["width"], s["ff"], s["heads"], s["kv_heads"], s["head_dim"]
    if arch == "llama":
        return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_act": "silu", "hidden_size": D, "intermediate_size": ff,
                "num_hidden_layers": n, "num_attention_heads": H, "num_key_value_heads": G, "head_dim": hd, "vocab_size": VOCAB,
                "max_position_embeddings": 131072, "rope_theta": 500000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": s["tied"],
                "rope_scaling": {"rope_type": "llama3", "factor": s["factor"], "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                                 "original_max_position_embeddings": 8192}}
    half, rot, lh = max(H // 2, 1), hd // 2, D // 128
    decay = [1.0 - 2.0 ** (-5 - 3 * i / max(1, lh - 1)) for i in range(lh)]
    dense = {"ff": ff, "kind": "dense"}
    latent = {"dim": hd, "heads": half, "kv_rank": min(512, D // 4), "scale": hd ** -0.5, "vdim": hd}
    experts = {"experts": 8, "top": 2}
    ssm = {"heads": D // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
    rms = {"norm": {"eps": 1e-6}, "vocab": VOCAB, "width": D}
    if arch == "nipadra":
        light = {"type": "lightning", "mixer": {"heads": lh, "dim": 128, "vdim": 128, "decay": decay}, "mlp": dense}
        both = {"type": "parallel", "mlp": dense, "mixer": {
            "left": {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "mask": {"size": 1024}, "rot": {"base": 500000.0, "dims": hd},
                     "scale": hd ** -0.5}, "right": ssm, "left_scale": 0.5, "right_scale": 0.5}}
        return dict(rms, architecture="Nipadra", postln_alpha=2.0, layers=[both if i % 4 == 2 else light for i in range(n)])
    if arch == "gekupel":
        lat = dict(latent, mask={"size": 1024}, q_rank=3 * D // 8, rot_dim=rot, rot={"base": 500000.0, "dims": rot}, scale=(hd + rot) ** -0.5)
        lat2 = dict(lat, rot={"base": 500000.0, "dims": rot, "scaling": {"factor": 4.0, "fast": 32.0, "original": 8192, "slow": 1.0}})
        att = {"dim": hd, "heads": H, "kv_heads": G, "mask": {"size": 1024}, "scale": hd ** -0.5, "vdim": hd}
        moe = {"expert": {"ff": ff // 2}, "kind": "moe", "router": experts}
        kinds = [("latent_attention_2", lat2, dense), ("attention", att, moe), ("latent_attention", lat, moe), ("attention", att, moe)]
        return dict(rms, architecture="Gekupel", embedding={"scale": 1.0},
                    layers=[{"type": t, "mixer": m, "mlp": f} for t, m, f in (kinds[i % 4] for i in range(n))])
    if arch == "pinorax":
        moe = {"expert": {"ff": 3 * ff // 8, "limit": 7.0}, "kind": "moe", "router": experts, "shared": {"ff": ff // 4, "limit": 7.0}}
        return dict(rms, architecture="Pinorax", logit_softcap=30.0, max_positions=_positions(case), residual_mult=0.5,
                    layers=[{"type": "latent_attention", "mixer": latent, "mlp": moe if i % 4 else dense} for i in range(n)])
    if arch == "fovezen":
        par = {"left": {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "mask": {"size": 1024}, "conv": 3, "softcap": 30.0, "scale": hd ** -0.5},
               "right": {"heads": D // 128, "dim": 64, "vdim": 128, "tau": 16.0, "rank": 16}}
        att = {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "scale": hd ** -0.5,
               "rot": {"base": 500000.0, "dims": rot, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        kinds = [("parallel", par), ("attention", att), ("mamba2", ssm), ("parallel", par)]
        return dict(rms, architecture="Fovezen", streams=2, logit_scale=0.5,
                    layers=[{"type": t, "mixer": m, "mlp": dict(dense, limit=7.0)} for t, m in (kinds[i % 4] for i in range(n))])
    if arch == "mimolix":
        moe = {"expert": {"ff": 9 * ff // 16}, "kind": "moe", "router": dict(experts, scale=2.0), "shared": {"ff": 3 * ff // 8}}
        delta = {"conv": 4, "dim": 128, "heads": lh, "kv_heads": max(D // 256, 1), "vdim": 128}
        att = {"diff": 0.5, "dim": hd // 2, "heads": half, "kv_heads": max(H // 8, 1), "q_temp": {"coef": 0.2, "every": 4096},
               "scale": (hd // 2) ** -0.5, "vdim": hd}
        kinds = [("delta", delta), ("attention", att), ("delta", delta), ("delta", delta)]
        return dict(rms, architecture="Mimolix", embedding={"scale": 3.0}, residual_mult=0.5, loop={"start": 0, "stop": n, "times": 1},
                    layers=[{"type": t, "mixer": m, "mlp": moe} for t, m in (kinds[i % 4] for i in range(n))])
    ret = {"heads": lh, "dim": 128, "vdim": 128, "decay": decay}
    att = {"heads": H, "kv_heads": G, "dim": hd, "vdim": hd, "scale": hd ** -0.5,
           "rot": {"base": 500000.0, "dims": hd, "scaling": {"factor": 4.0}}}
    lat = dict(latent, rot_dim=rot, scale=(hd + rot) ** -0.5,
               rot={"base": 500000.0, "dims": rot, "scaling": {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}})
    moe = {"expert": {"ff": 3 * ff // 8}, "kind": "moe", "router": experts, "shared": {"ff": ff // 4}}
    kinds = [("retention", ret, {"ff": 3 * ff // 2, "kind": "dense"}), ("attention", att, moe), ("latent_attention", lat, moe), ("retention", ret, moe)]
    return dict(rms, architecture="Kidarax", logit_scale=0.5, layers=[{"type": t, "mixer": m, "mlp": f} for t, m, f in (kinds[i % 4] for i in range(n))])


def _positions(case):
    """Context length of the engine: room for the longest request, a multiple of 64."""
    longest = max(_lengths(case)) + case["new"] + case["tokens"]
    return (longest + 63) // 64 * 64


# ---------------------------------------------------------------------------------------------------- inputs
def _generator(seed, name):
    return torch.Generator("cuda").manual_seed((zlib.crc32(name.encode()) << 20) + 1000003 * seed + 17)


def _plan(case):
    from geneinfer_b200.config import parse_config
    arch, cfg = parse_config(config_of(case))
    return cfg, arch.weight_plan(cfg)


def _weights(case, seed):
    """The checkpoint's tensors by name, on the device. Matrices N(0, 0.02) as the benchmark draws them, but for what random
    numbers would leave unlike a trained model: products that end a branch are smaller the deeper the model, a tied head
    gives logits of which few tokens hold the probability, and a token's embedding holds the directions of the two experts
    its routers look for (routers that decide, and not ties)."""
    arch, dtype = case["arch"], getattr(torch, case["dtype"])
    _, plan = _plan(case)
    D = SIZES[case["size"]]["width"]
    ways = (torch.rand(8, D, generator=_generator(seed, "experts"), device="cuda") < 0.5).float().mul_(2).sub_(1)
    out = {}
    for rule in plan.rules:
        name, init, shape, g = rule.name, rule.init, rule.shape, _generator(seed, rule.name)
        if rule.kind == "table":
            out[name] = torch.rand(shape[0], init[1], generator=g, device="cuda").argsort(1)[:, :shape[1]].to(torch.int32).contiguous()
            continue
        if init is not None and init[0] == "uniform":
            out[name] = torch.rand(shape, generator=g, device="cuda").mul_(init[2] - init[1]).add_(init[1]).to(dtype)
            continue
        mean, std = (init if init is not None else (1.0, 0.02) if rule.kind == "vector" else (0.0, 0.02))
        if arch == "llama" and name.endswith(("o_proj.weight", "down_proj.weight")):
            std = 0.02 / case["layers"] ** 0.5
        if name in ("embed", "model.embed_tokens.weight"):
            std = 0.5 if arch in DESIGNS[:-1] else 0.1
        t = torch.randn(shape, generator=g, device="cuda").mul_(std).add_(mean)
        if name == "embed" and arch in ROUTED:
            two = torch.rand(shape[0], 8, generator=g, device="cuda").argsort(1)
            t.add_(ways[two[:, 0]], alpha=std).add_(ways[two[:, 1]], alpha=0.8 * std)
        if name.endswith("mlp.router"):
            t = ways * (0.1 / D ** 0.5) + 0.05 * t
        if name == "loop.in":           # the embedding's output goes on beside the stream
            t.mul_(0.2).add_(torch.eye(D, device="cuda").repeat(1, 2), alpha=0.5)
        out[name] = t.to(dtype)
    return out


def _tokens(case, seed):
    """Token ids of every request: the cached ones or its prompt, then the ``new`` ones; last of all the portion (prefill, mixed)."""
    g = torch.Generator().manual_seed(7919 * seed + 3)
    lengths = [] if case["mode"] == "prefill" else [n + case["new"] for n in _lengths(case)]
    if case["tokens"]:
        lengths.append(case["tokens"])
    return [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in lengths]


def _draws(case, seed):
    """How each request of a sampled case draws: (temperature, top_k, top_p) and its random numbers, one per token."""
    g = torch.Generator().manual_seed(104729 * seed + 5)
    kinds = [(0.0, 0, 1.0), (0.8, 0, 1.0), (0.7, 40, 1.0), (1.0, 0, 0.9), (0.9, 50, 0.95)]
    return [(kinds[i % 5], torch.rand(case["new"], generator=g).tolist()) for i in range(case["requests"])]


def prepare(case, seed):
    from geneinfer_b200 import SamplingParams, StepEngine, StepEntry
    from geneinfer_b200.parts import DecoderModel
    from geneinfer_b200.sampling.device import DeviceSampler
    cfg, plan = _plan(case)
    device, positions = torch.device("cuda:0"), _positions(case)
    model = DecoderModel(cfg.model_spec(), plan.assemble(_weights(case, seed)), getattr(torch, case["dtype"]), device, positions)
    tokens, lengths, mode = _tokens(case, seed), _lengths(case), case["mode"]
    requests = len(tokens)
    pages = sum((len(t) + PAGE - 1) // PAGE for t in tokens) + requests
    engine = StepEngine(model, page_size=PAGE, n_pages=pages, max_requests=requests, max_step_tokens=STEP_TOKENS, max_logit_rows=requests)
    state = {"engine": engine, "entry": StepEntry, "case": case, "tokens": tokens, "lengths": lengths}
    if mode in ("decode", "mixed"):          # the texts so far are in the cache
        for i, n in enumerate(lengths):
            engine.open(i)
            for at in range(0, n, STEP_TOKENS):
                engine.step([StepEntry(i, tokens[i][at:min(n, at + STEP_TOKENS)])])
    if mode == "sampled":
        state["sampler"] = DeviceSampler(VOCAB, device, ids=engine.feedback)
        draws = _draws(case, seed)
        state["params"] = [SamplingParams(*kind) for kind, _ in draws]
        state["uniforms"] = [[u[t] for _, u in draws] for t in range(case["new"])]
    engine.check_status()
    return state


# ---------------------------------------------------------------------------------------------------- one pass
def run(state):
    engine, entry, case, tokens, lengths = (state[k] for k in ("engine", "entry", "case", "tokens", "lengths"))
    mode = case["mode"]
    if mode in ("decode", "mixed"):          # every request's next token; the portion's last row is wanted too
        for i, n in enumerate(lengths):
            engine.truncate(i, n)
        step = [entry(i, tokens[i][n:], [0]) for i, n in enumerate(lengths)]
        if mode == "decode":
            return engine.step(step)
        engine.open("portion")
        logits = engine.step(step + [entry("portion", tokens[-1], [case["tokens"] - 1])])
        engine.close("portion")
        return logits
    if mode == "prefill":
        engine.open("prompt")
        for at in range(0, case["tokens"], STEP_TOKENS):
            portion = tokens[0][at:at + STEP_TOKENS]
            last = at + len(portion) == case["tokens"]
            logits = engine.step([entry("prompt", portion, [len(portion) - 1] if last else [])])
        engine.close("prompt")
        return logits
    keys = range(len(lengths))
    for i in keys:
        engine.open(i)
    logits = engine.step([entry(i, tokens[i][:n], [n - 1]) for i, n in enumerate(lengths)])
    out = {"prompt": logits.clone()}
    if mode == "sampled":                    # each token drawn on the device, and read from there by the next step
        ids = []
        for uniforms in state["uniforms"]:
            state["sampler"].sample_async(logits, state["params"], uniforms)
            ids.append(engine.feedback[:len(keys)].clone())
            logits = engine.step([entry(i, [-(i + 1)], [0]) for i in keys])
        out["ids"], out["last"] = torch.stack(ids), logits.clone()
    else:
        decoded = []
        for t in range(case["new"]):
            decoded.append(engine.step([entry(i, [tokens[i][lengths[i] + t]], [0]) for i in keys]).clone())
        out["decoded"] = torch.stack(decoded)
    for i in keys:
        engine.close(i)
    return out


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _mixers(config):
    """(kind, constants) of every mixer, those beside each other one by one."""
    out = []
    for layer in config["layers"]:
        m = layer["mixer"]
        out += [("attention", m["left"]), ("state", m["right"])] if layer["type"] == "parallel" else [(layer["type"], m)]
    return out


def _mixer_cost(kind, m):
    """(cached values a position, flops per query and key, positions seen at most, values of the state, flops a token of the state)."""
    if kind == "attention" or kind.startswith("latent"):
        span = (m.get("mask") or {}).get("size", 1 << 30)
        maps = 2 if "diff" in m else 1
        if "kv_rank" in m:
            return m["kv_rank"] + m.get("rot_dim", 0), 2 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"]), span, 0, 0
        return m["kv_heads"] * (maps * m["dim"] + m["vdim"]), 2 * maps * m["heads"] * (m["dim"] + m["vdim"]), span, 0, 0
    values = m["heads"] * m.get("state", m.get("dim")) * m["vdim"]
    return 0, 0, 0, values, values * (6 if kind == "delta" else 4)


def _step_work(case, mixers, rules, steps):
    """Bytes and flops of steps, each a list of (cached, new tokens) per request and the number of wanted rows."""
    elt = 4 if case["dtype"] == "float32" else 2
    D, nbytes, flops = SIZES[case["size"]]["width"], 0.0, 0.0
    body = sum(math.prod(r.shape) for r in rules if r.kind != "table" and r.name not in ("embed", "model.embed_tokens.weight", "pos", "head", "lm_head.weight")
               and not re.search(r"mlp\.e\d+\.", r.name))
    expert = sum(math.prod(r.shape) for r in rules if re.search(r"mlp\.e\d+\.", r.name))
    for requests, wanted in steps:
        T = sum(n for _, n in requests)
        used = 1.0 - 0.75 ** T                     # the share of eight experts that T tokens with two each reach
        nbytes += elt * (body + used * expert + T * D) + (elt * VOCAB * D + 4 * wanted * VOCAB if wanted else 0)
        flops += 2.0 * T * (body + expert / 4) + 2.0 * wanted * VOCAB * D
        for kind, m in mixers:
            width, pair, span, values, each = _mixer_cost(kind, m)
            for cached, n in requests:
                seen = min(cached, span)
                nbytes += elt * width * (seen + n) + 8 * values
                flops += pair * sum(min(span, cached + i + 1) for i in range(n)) + each * n
    return {"bytes": nbytes, "flops": flops}


def work(case):
    config, lengths = config_of(case), _lengths(case)
    if case["arch"] == "llama":
        s = SIZES[case["size"]]
        mixers = [("attention", {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": s["head_dim"], "vdim": s["head_dim"]})] * case["layers"]
    else:
        mixers = _mixers(config)
    _, plan = _plan(case)
    mode, new = case["mode"], case["new"]
    if mode == "prefill":
        parts = [(at, min(STEP_TOKENS, case["tokens"] - at)) for at in range(0, case["tokens"], STEP_TOKENS)]
        steps = [([p], int(p is parts[-1])) for p in parts]
    elif mode in ("decode", "mixed"):
        steps = [([(n, 1) for n in lengths] + ([(0, case["tokens"])] if case["tokens"] else []), len(lengths) + (mode == "mixed"))]
    else:
        steps = [([(0, n) for n in lengths], len(lengths))] + [([(n + t, 1) for n in lengths], len(lengths)) for t in range(new)]
    return _step_work(case, mixers, plan.rules, steps)


# About four times what the logits were seen to be off from 64 bits (a whole model in bfloat16: 0.012 at 16 layers).
_OFF = {"llama": 0.03, "nipadra": 0.016, "gekupel": 0.016, "pinorax": 0.02, "fovezen": 0.03, "mimolix": 0.016, "kidarax": 0.004}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.01}
    rel = _OFF[case["arch"]]
    return {"rel": rel, "max": 10 * rel}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
F = torch.float64


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _softplus(z):
    return torch.nn.functional.softplus(z, threshold=1e9)


def _attend(q, k, v, scale, window=None, block=None, slope=None, sink=None, cap=None):
    """Causal attention of one sequence: q [n, H, d], k [n, G, d], v [n, G, dv]. ``window`` and ``block`` limit what a query sees,
    ``slope`` [H] takes off the distance, ``sink`` [H] stands in the denominator, ``cap`` bounds the scores."""
    n, H, _ = q.shape
    per = H // k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=F, device=q.device)
    at = torch.arange(n, device=q.device)
    rows = max(1, (1 << 27) // max(1, n))
    for a in range(0, n, rows):
        i = at[a:a + rows, None]
        j = at[None, :min(n, a + rows)]
        seen = j <= i
        if window:
            seen &= i - j < window
        if block:
            seen &= torch.div(i, block, rounding_mode="floor") == torch.div(j, block, rounding_mode="floor")
        for h in range(H):
            s = q[a:a + rows, h] @ k[:j.shape[1], h // per].T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            if slope is not None:
                s = s - slope[h] * (i - j)
            s.masked_fill_(~seen, -math.inf)
            top = s.amax(1, keepdim=True)
            if sink is not None:
                top = torch.maximum(top, sink[h])
            e = torch.exp_(s - top)
            total = e.sum(1, keepdim=True)
            if sink is not None:
                total = total + torch.exp(sink[h] - top)
            out[a:a + rows, h] = (e / total) @ v[:j.shape[1], h // per]
    return out


def _frequencies(rot):
    """(frequency of each pair, factor on cosine and sine) of a rotation with one of the designs' long-context scalings."""
    dims, base, s = rot["dims"], float(rot["base"]), rot.get("scaling")
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F) / dims)
    if not s:
        return f, 1.0
    factor = float(s["factor"])
    if "low" in s:                            # by wavelength: short ones stay, long ones are divided, between them a blend
        share = ((s["original"] * f / (2 * math.pi) - s["low"]) / (s["high"] - s["low"])).clamp(0, 1)
        return (1 - share) * f / factor + share * f, 1.0
    if "original" not in s:
        return f / factor, 1.0
    place = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(place(s["fast"])), 0), min(math.ceil(place(s["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / factor * ramp + f * (1 - ramp), 0.1 * math.log(factor) + 1.0


def _rotate(x, rot, interleaved):
    """x [n, heads, d] at positions 0 .. n-1: the first ``dims`` dimensions turn in pairs (neighbours, or halves apart)."""
    f, by = _frequencies(rot)
    angle = torch.arange(x.shape[0], dtype=F, device=x.device)[:, None, None] * f.to(x.device)
    c, s, dims = torch.cos(angle) * by, torch.sin(angle) * by, rot["dims"]
    out = x.clone()
    one, two = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., one] = x[..., one] * c - x[..., two] * s
    out[..., two] = x[..., two] * c + x[..., one] * s
    return out


def _scan(q, k, v, fade):
    """S <- fade S + k v^T, o = S^T q over the tokens. q, k [n, H, d], v [n, H, dv], fade broadcastable to [n, H, d]."""
    n, H, d = q.shape
    S = torch.zeros(H, d, v.shape[2], dtype=F, device=q.device)
    fade = fade.expand(n, H, d)
    out = torch.empty_like(v)
    for t in range(n):
        S.mul_(fade[t, :, :, None]).addcmul_(k[t, :, :, None], v[t, :, None, :])
        out[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
    return out


def _delta(q, k, v, beta, fade):
    """The gated delta rule: fade, correct what the key reads, read out."""
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S.mul_(fade[t, :, None, None])
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None, :], S)[:, 0])
        S.addcmul_(k[t, :, :, None], u[:, None, :])
        out[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
    return out


def _conv(u, w, bias=None):
    """A short causal filter per channel. u [n, C], w [C, taps] with the newest tap last."""
    taps = w.shape[1]
    pad = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    y = sum(pad[j:j + u.shape[0]] * w[:, j] for j in range(taps))
    return y if bias is None else y + bias


class _Weights:
    """Tensors below a prefix, widened when they are read."""

    def __init__(self, tensors, prefix=""):
        self.tensors, self.prefix = tensors, prefix

    def __call__(self, name):
        t = self.tensors[self.prefix + name]
        return t if t.dtype == torch.int32 else t.to(F)

    def __contains__(self, name):
        return self.prefix + name in self.tensors

    def at(self, prefix):
        return _Weights(self.tensors, self.prefix + prefix)


def _ssm(h, w, m, eps):
    """State-space mixer ahead of its output product: convolved inputs, one decay a head and token."""
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    n, inner = h.shape[0], m["heads"] * m["vdim"]
    z, xbc, step = (h @ w("in").T).split([inner, inner + 2 * G * N, H], 1)
    xs, B, C = _silu(_conv(xbc, w("conv"), w("conv.b"))).split([inner, G * N, G * N], 1)
    xs = xs.reshape(n, H, P)
    B, C = (t.reshape(n, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    step = _softplus(step + w("dt_bias"))
    y = _scan(C, step[:, :, None] * B, xs, torch.exp(-torch.exp(w("A_log")) * step)[:, :, None]) + w("D")[:, None] * xs
    y = (y.reshape(n, inner) * _silu(z)).reshape(n, m["norm_groups"], -1)
    return _unit(y, eps).reshape(n, inner) * w("norm")


def _nipadra(h, w, kind, m, eps):
    n = h.shape[0]
    if kind == "lightning":
        H = m["heads"]
        q, k, v = (_silu(h @ w(c).T).reshape(n, H, -1) for c in "qkv")
        fade = torch.tensor(m["decay"], dtype=F, device=h.device)[None, :, None]
        return (_unit(_scan(q, k, v, fade).reshape(n, -1), eps) * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T
    a, l = m["left"], w.at("left.")
    q, k = (h @ l("q").T).reshape(n, a["heads"], -1), (h @ l("k").T).reshape(n, a["kv_heads"], -1)
    v = k
    q, k = (_rotate(_unit(t, eps) * l(c + ".norm"), a["rot"], True) for t, c in ((q, "q"), (k, "k")))
    zero = torch.zeros(a["heads"], dtype=F, device=h.device)
    o = _attend(q, k, v, a["scale"], window=a["mask"]["size"], sink=zero) * torch.sigmoid(h @ l("g").T)[:, :, None]
    r = w.at("right.")
    return m["left_scale"] * (o.reshape(n, -1) @ l("o").T) + m["right_scale"] * (_ssm(h, r, m["right"], eps) @ r("o").T)


def _gekupel(h, w, kind, m, eps):
    n, H = h.shape[0], m["heads"]
    if kind == "attention":
        q, k = (_unit((h @ w(c).T).reshape(n, g, -1), eps) for c, g in (("q", H), ("k", m["kv_heads"])))
        v = (h @ w("v").T).reshape(n, m["kv_heads"], -1)
        slope = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=F, device=h.device) / H)
        return _attend(q, k, v, m["scale"], block=m["mask"]["size"], slope=slope, sink=w("sink")).reshape(n, -1) @ w("o").T
    d, rank = m["dim"], m["kv_rank"]
    rot = m["rot"] if kind.endswith("_2") else {k: v for k, v in m["rot"].items() if k != "scaling"}
    q = (_unit(h @ w("dq").T, eps) * w("dq.norm") @ w("uq").T).reshape(n, H, -1)
    down = h @ w("dkv").T
    c = _unit(down[:, :rank], eps) * w("dkv.norm")
    kr = _rotate(down[:, None, rank:], rot, True).expand(n, H, -1)
    k = torch.cat([(c @ w("uk").T).reshape(n, H, d), kr], 2)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], rot, True)], 2)
    v = (c @ w("uv").T).reshape(n, H, -1)
    sink = w("sink") if kind.endswith("_2") else None
    return _attend(q, k, v, m["scale"], window=m["mask"]["size"], sink=sink).reshape(n, -1) @ w("o").T


def _pinorax(h, w, kind, m, eps):
    n, H = h.shape[0], m["heads"]
    q = (h @ w("q").T).reshape(n, H, -1)
    c = _unit(h @ w("dkv").T, eps) * w("dkv.norm")
    k, v = (c @ w("uk").T).reshape(n, H, -1), (c @ w("uv").T).reshape(n, H, -1)
    o = _attend(q, k, v, m["scale"], sink=w("sink")).reshape(n, -1)
    return (o * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _fovezen(h, w, kind, m, eps):
    n = h.shape[0]
    if kind == "mamba2":
        return _ssm(h, w, m, eps) @ w("o").T
    if kind == "attention":
        H, G = m["heads"], m["kv_heads"]
        q, k = ((_unit(h @ w(c).T, eps) * w(c + ".norm")).reshape(n, g, -1) for c, g in (("q", H), ("k", G)))
        q, k = _rotate(q, m["rot"], False), _rotate(k, m["rot"], False)
        return _attend(q, k, (h @ w("v").T).reshape(n, G, -1), m["scale"]).reshape(n, -1) @ w("o").T
    a, l = m["left"], w.at("left.")
    q, k, v = (_conv(h @ l(c).T, l(c + ".conv")).reshape(n, a["heads"] if c == "q" else a["kv_heads"], -1) for c in "qkv")
    q, k = _unit(q, eps) * l("q.norm"), _unit(k, eps) * l("k.norm")
    left = _attend(q, k, v, a["scale"], window=a["mask"]["size"], cap=a["softcap"]).reshape(n, -1) @ l("o").T
    b, r = m["right"], w.at("right.")
    q, k, v = ((h @ r(c).T).reshape(n, b["heads"], -1) for c in "qkv")
    fade = torch.exp(-_softplus(-((h @ r("a1").T) @ r("a2").T + r("a2.b"))) / b["tau"]).reshape(n, b["heads"], -1)
    o = _unit(_scan(q * b["dim"] ** -0.5, k, v, fade), eps) * r("norm")
    right = (o.reshape(n, -1) * _silu(h @ r("g").T)) @ r("o").T
    return 0.5 * (_unit(left, eps) * w("left.out") + _unit(right, eps) * w("right.out"))


def _mimolix(h, w, kind, m, eps):
    n, H, G = h.shape[0], m["heads"], m["kv_heads"]
    if kind == "attention":
        q, k = (_unit((h @ w(c).T).reshape(n, g, 2, -1), eps) * w(c + ".norm") for c, g in (("q", H), ("k", G)))
        block = torch.floor(torch.arange(1, n + 1, dtype=F, device=h.device) / m["q_temp"]["every"])
        q = q * (1.0 + m["q_temp"]["coef"] * torch.log(block + 1.0))[:, None, None, None]
        v = (h @ w("v").T).reshape(n, G, -1)
        one, two = (_attend(q[:, :, i], k[:, :, i], v, m["scale"]) for i in (0, 1))
        weight = torch.exp((w("lq1") * w("lk1")).sum()) - torch.exp((w("lq2") * w("lk2")).sum()) + m["diff"]
        return (_unit(one - weight * two, eps) * (1.0 - m["diff"])).reshape(n, -1) @ w("o").T
    q, k, v = (_silu(_conv(h @ w(c).T, w(c + ".conv"))) for c in "qkv")
    q, k = (t.reshape(n, G, -1) for t in (q, k))
    q, k = ((t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for t in (q, k))
    beta = torch.sigmoid(h @ w("b").T)
    fade = torch.exp(-torch.exp(w("A_log")) * _softplus(h @ w("a").T + w("dt_bias")))
    o = _unit(_delta(q * m["dim"] ** -0.5, k, v.reshape(n, H, -1), beta, fade), eps) * w("norm")
    return (o.reshape(n, -1) * _silu(h @ w("g").T)) @ w("o").T


def _kidarax(h, w, kind, m, eps):
    n, H = h.shape[0], m["heads"]
    if kind == "retention":
        q, k, v = ((h @ w(c).T).reshape(n, H, -1) for c in "qkv")
        fade = torch.tensor(m["decay"], dtype=F, device=h.device)[None, :, None]
        o = _unit(_scan(q, k * m["dim"] ** -0.5, v, fade), eps).reshape(n, -1)
        return (o * _silu(h @ w("g").T)) @ w("o").T
    if kind == "attention":
        q, k, v = ((h @ w(c).T + w(c + ".b")).reshape(n, H if c == "q" else m["kv_heads"], -1) for c in "qkv")
        o = _attend(_rotate(q, m["rot"], False), _rotate(k, m["rot"], False), v, m["scale"]).reshape(n, -1)
        return (o * torch.sigmoid(h @ w("g").T)) @ w("o").T
    d, rank = m["dim"], m["kv_rank"]
    q = (h @ w("q").T).reshape(n, H, -1)
    down = h @ w("dkv").T
    c = _unit(down[:, :rank], eps) * w("dkv.norm")
    k = torch.cat([(c @ w("uk").T).reshape(n, H, d), _rotate(down[:, None, rank:], m["rot"], False).expand(n, H, -1)], 2)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"], False)], 2)
    o = _attend(q, k, (c @ w("uv").T).reshape(n, H, -1), m["scale"], sink=w("sink"))
    return (o * torch.sigmoid(h @ w("g").T)[:, :, None]).reshape(n, -1) @ w("o").T


def _llama(h, w, kind, m, eps):
    n = h.shape[0]
    q, k, v = ((h @ w(f"self_attn.{c}_proj.weight").T).reshape(n, m["heads"] if c == "q" else m["kv_heads"], -1) for c in "qkv")
    o = _attend(_rotate(q, m["rot"], False), _rotate(k, m["rot"], False), v, m["scale"])
    return o.reshape(n, -1) @ w("self_attn.o_proj.weight").T


def _expert(arch, w, x, limit):
    if arch == "mimolix":
        return torch.relu(x @ w("up").T).square() @ w("down").T
    g, u = x @ w("gate").T, x @ w("up").T
    if arch == "pinorax":
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w("down").T
    return (_silu(g) * u) @ w("down").T


def _feed_forward(arch, f, w, h, tokens):
    """The feed-forward of all requests' rows at once."""
    if f["kind"] == "dense":
        if arch == "kidarax":
            return torch.relu(h @ w("up").T).square() @ w("down").T
        g, u = h @ w("gate").T, h @ w("up").T
        if arch == "nipadra":
            return (torch.relu(g) * u) @ w("down").T
        if arch == "gekupel":
            return (torch.nn.functional.gelu(g, approximate="tanh") * u) @ w("down").T
        if arch == "pinorax":
            g, u = g + w("gate.b"), u + w("up.b")
            return (_silu(g) * u) @ w("down").T + w("down.b")
        g, u = g.clamp(max=f["limit"]), u.clamp(-f["limit"], f["limit"])
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w("down").T
    top = f["router"]["top"]
    if arch == "pinorax":
        ids = w("table")[tokens].long()
        share = torch.full(ids.shape, 1.0 / top, dtype=F, device=h.device)
    else:
        s = h @ w("router").T
        s = torch.softmax(s, -1) if arch == "mimolix" else torch.sigmoid(s)
        ids = torch.topk(s + w("correction") if arch == "gekupel" else s, top, -1).indices
        share = torch.gather(s, 1, ids)
        if arch == "mimolix":
            share = share / (share.sum(-1, keepdim=True) + 1e-20) * f["router"]["scale"]
    y = torch.zeros_like(h)
    limit = f["expert"].get("limit")
    for e in range(f["router"]["experts"]):
        t, c = torch.nonzero(ids == e, as_tuple=True)
        if len(t):
            by = share[t, c][:, None]
            if arch == "kidarax":
                y[t] += _expert(arch, w.at(f"e{e}."), by * h[t], limit)
            else:
                y[t] += by * _expert(arch, w.at(f"e{e}."), h[t], limit)
    if f.get("shared"):
        z = _expert(arch, w.at("shared."), h, f["shared"].get("limit"))
        y = y + (torch.sigmoid(h @ w("shared.sg").T) * z if arch == "kidarax" else z)
    return y


def _forward(case, tensors, texts, wanted):
    """Logits [wanted, vocab] of whole texts; ``wanted``: (text, place) pairs."""
    arch, config, w = case["arch"], config_of(case), _Weights(tensors)
    lengths = [len(t) for t in texts]
    tokens = torch.tensor([t for text in texts for t in text], device="cuda")
    starts = [sum(lengths[:i]) for i in range(len(texts))]
    rows = torch.tensor([starts[i] + at for i, at in wanted], device="cuda")

    def mixed(mixer, h, part, kind, m, eps):
        return torch.cat([mixer(t, part, kind, m, eps) for t in h.split(lengths)])

    if arch == "llama":
        s, r, eps = SIZES[case["size"]], config["rope_scaling"], config["rms_norm_eps"]
        m = {"heads": s["heads"], "kv_heads": s["kv_heads"], "scale": s["head_dim"] ** -0.5,
             "rot": {"base": config["rope_theta"], "dims": s["head_dim"], "scaling": {
                 "factor": r["factor"], "low": r["low_freq_factor"], "high": r["high_freq_factor"], "original": r["original_max_position_embeddings"]}}}
        x = tensors["model.embed_tokens.weight"][tokens].to(F)
        for i in range(case["layers"]):
            l = w.at(f"model.layers.{i}.")
            x = x + mixed(_llama, _unit(x, eps) * l("input_layernorm.weight"), l, "attention", m, eps)
            h = _unit(x, eps) * l("post_attention_layernorm.weight")
            for a in range(0, h.shape[0], 16384):
                part = h[a:a + 16384]
                x[a:a + 16384] += (_silu(part @ l("mlp.gate_proj.weight").T) * (part @ l("mlp.up_proj.weight").T)) @ l("mlp.down_proj.weight").T
        head = tensors["lm_head.weight"] if "lm_head.weight" in tensors else tensors["model.embed_tokens.weight"]
        return (_unit(x[rows], eps) * w("model.norm.weight")) @ head.to(F).T

    eps = config["norm"]["eps"]
    mixer = {"nipadra": _nipadra, "gekupel": _gekupel, "pinorax": _pinorax, "fovezen": _fovezen, "mimolix": _mimolix, "kidarax": _kidarax}[arch]
    x = tensors["embed"][tokens].to(F)
    if arch == "pinorax":
        x = x + w("pos")[torch.cat([torch.arange(n, device="cuda") for n in lengths])]
        results = [x]
    if arch == "mimolix":
        x = x * config["embedding"]["scale"]
        x = torch.cat([x, x], 1) @ w("loop.in").T              # one pass: the stream ahead of it is the embedding's output
    if arch == "fovezen":
        x = x[None].repeat(config["streams"], 1, 1)

    def tanh_norm(name, v):
        return torch.tanh(w(name + ".alpha") * v) * w(name) + w(name + ".b")

    for i, layer in enumerate(config["layers"]):
        p, l = f"l{i}.", w.at(f"l{i}.")
        mix = lambda h: mixed(mixer, h, l.at("mix."), layer["type"], layer["mixer"], eps)  # noqa: E731
        ff = lambda h: _feed_forward(arch, layer["mlp"], l.at("mlp."), h, tokens)  # noqa: E731
        if arch == "nipadra":
            for f, norm in ((mix, "norm1"), (ff, "norm2")):
                x = _unit(config["postln_alpha"] * x + f(x), eps) * (1.0 + l(norm))
        elif arch == "gekupel":
            for f, norm in ((mix, "norm1"), (ff, "norm2")):
                x = x + _unit(f(x), eps) * l(norm)
        elif arch == "pinorax":
            h = _unit(x, eps) * l("norm1")
            results.append(x + config["residual_mult"] * (mix(h) + ff(h)))
            x = sum(a * r for a, r in zip(l("dwa"), results))
        elif arch == "fovezen":
            for f, norm, hc in ((mix, "norm1", l.at("hc1.")), (ff, "norm2", l.at("hc2."))):
                y = f(_unit(torch.einsum("s,std->td", hc("in"), x), eps) * (1.0 + l(norm)))
                x = torch.einsum("sr,std->rtd", hc("mix"), x) + hc("out")[:, None, None] * y
        elif arch == "mimolix":
            d = x - x.mean(-1, keepdim=True)
            h = _unit(d, eps) * l("norm1") + l("norm1.b")
            x = x + config["residual_mult"] * (mix(h) + ff(h))
        else:
            x = x + tanh_norm(p + "norm1b", mix(tanh_norm(p + "norm1", x)))
            x = x + tanh_norm(p + "norm2b", ff(tanh_norm(p + "norm2", x)))
    if arch == "fovezen":
        x = x.sum(0)
    x = x[rows]
    if arch in ("nipadra", "fovezen"):
        x = _unit(x, eps) * (1.0 + w("final.norm"))
    elif arch == "mimolix":
        x = _unit(x - x.mean(-1, keepdim=True), eps) * w("final.norm") + w("final.norm.b")
    elif arch == "kidarax":
        x = tanh_norm("final.norm", x)
    else:
        x = _unit(x, eps) * w("final.norm")
    logits = x @ w("head" if "head" in w else "embed").T * config.get("logit_scale", 1.0)
    cap = config.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits


def _pick(logits, kind, u):
    """One token of a row of logits: the largest, or drawn by ``u`` from the probabilities that the filters leave, in the order of
    the probabilities where a filter is on and of the ids where none is."""
    temperature, top_k, top_p = kind
    if temperature <= 0:
        return int(logits.argmax())
    p = torch.softmax(logits / temperature, 0)
    order = torch.arange(p.numel(), device=p.device)
    if top_k or top_p < 1.0:
        p, order = torch.sort(p, descending=True, stable=True)
        if top_k:
            p = p[:top_k]
        if top_p < 1.0:
            total = torch.cumsum(p, 0)
            p = p[:int((total < top_p * total[-1]).sum()) + 1]
    at = int((torch.cumsum(p, 0) <= u * p.sum()).sum())
    return int(order[min(at, p.numel() - 1)])


def exact(case, seed):
    tensors, tokens, lengths, new = _weights(case, seed), _tokens(case, seed), _lengths(case), case["new"]
    mode = case["mode"]
    if mode in ("decode", "mixed", "prefill"):
        return _forward(case, tensors, tokens, [(i, len(t) - 1) for i, t in enumerate(tokens)])
    if mode == "sampled":
        draws = _draws(case, seed)
        texts = [t[:n] for t, n in zip(tokens, lengths)]
        prompt = logits = _forward(case, tensors, texts, [(i, n - 1) for i, n in enumerate(lengths)])
        for t in range(new):
            for i, (kind, u) in enumerate(draws):
                texts[i].append(_pick(logits[i], kind, u[t]))
            logits = _forward(case, tensors, texts, [(i, len(x) - 1) for i, x in enumerate(texts)])
        ids = torch.tensor([x[n:] for x, n in zip(texts, lengths)]).T.to(torch.int32)
        return {"prompt": prompt, "ids": ids, "last": logits}
    logits = _forward(case, tensors, tokens, [(i, n - 1 + t) for t in range(new + 1) for i, n in enumerate(lengths)])
    logits = logits.view(new + 1, len(lengths), VOCAB)
    return {"prompt": logits[0], "decoded": logits[1:]}
