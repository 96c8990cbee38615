"""The workloads whose time and results are measured.

A case is one pass of a user's program through the framework: a batch of prompts in one ``Engine.step`` (logits at every
prompt's last token, or at every token where prompts are scored), then ``steps`` steps of one token a sequence, then the
slots are closed; or one call of the sampler on a batch of logits.  Models are the shapes that the repository's own
configurations, tests and benchmark use, with random weights; the larger ones keep a few of their layers, each of the real
size, so that a pass stays short.  ``exact`` restates every model in 64 bits with torch alone.

Fields of a case: ``kind`` "model" or "sample".  Models: ``model`` and ``layers`` (a shape of ``_config``), ``dtype``,
``batch`` prompts of ``shortest`` to ``longest`` tokens, ``scored`` (logits of every prompt token), ``steps`` single-token
steps, ``generate`` (the steps are fed with the ids that the sampler chose, on the device, as the generation loop does; else
with given ids, as trace replay and scoring do).  Sampler: ``rows``, ``vocab``, ``temperature``, ``top_k``, ``top_p``,
``penalty``.
"""
import math
import random

import torch

import xeno_rt_b200 as xrt
from xeno_rt_b200.cache import BLOCK_TOKENS, Cache
from xeno_rt_b200.sampling import Sampler, SamplerConfig

DEVICE = "cuda:0"


# ----------------------------------------------------------------------------- models
def _dense(arch, width, heads, kv_heads, head_dim, inner, vocab, theta, eps, tied=False, positions=16384):
    return {"architectures": [arch], "vocab_size": vocab, "max_position_embeddings": positions, "hidden_size": width,
            "intermediate_size": inner, "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": head_dim,
            "rope_theta": theta, "rms_norm_eps": eps, "tie_word_embeddings": tied}


_LLAMA, _QWEN3 = "LlamaForCausalLM", "Qwen3ForCausalLM"
_DENSE = {
    "tiny-llama": (2, _dense(_LLAMA, 64, 4, 2, 16, 176, 256, 10000.0, 1e-5, positions=128)),
    "tiny-qwen3": (3, _dense(_QWEN3, 96, 6, 2, 32, 160, 320, 1e6, 1e-6, tied=True, positions=256)),
    "llama-2k": (8, _dense(_LLAMA, 2048, 16, 4, 128, 8192, 32000, 500000.0, 1e-5)),
    "llama3-8b": (32, _dense(_LLAMA, 4096, 32, 8, 128, 14336, 128256, 500000.0, 1e-5)),
    "qwen3-8b": (36, _dense(_QWEN3, 4096, 32, 8, 128, 12288, 151936, 1e6, 1e-6)),
    "qwen3-32b": (64, _dense(_QWEN3, 5120, 64, 8, 128, 25600, 151936, 1e6, 1e-6)),
}
_SIZES = {"2k": (2048, 16, 4, 128, 8192, 32000), "4k": (4096, 32, 8, 128, 14336, 128256)}


def _config(case):
    """config.json of the case's model; the designs beside the dense decoder as the benchmark lays them out."""
    name, n = case["model"], case["layers"]
    if name in _DENSE:
        return dict(_DENSE[name][1], num_hidden_layers=n)
    design, size = name.split("-")
    width, heads, kv, dim, inner, vocab = _SIZES[size]
    if design == "givopel":
        rot = {"base": 500000.0, "dims": dim, "scaling": {"factor": 4.0, "original": 4096, "fast": 16.0, "slow": 2.0}}
        mlp = {"kind": "dense", "ff": inner}
        kinds = [{"type": "parallel", "mlp": mlp, "mixer": {
                     "left": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "rot": rot},
                     "right": {"heads": heads, "kv_heads": heads // 2, "dim": dim, "vdim": dim, "conv": 4, "decay_rank": 64,
                               "gate_rank": 64}}},
                 {"type": "gla", "mlp": mlp,
                  "mixer": {"heads": heads // 2, "dim": dim, "vdim": 2 * dim, "tau": 8.0, "decay_rank": 64}}]
        return {"architecture": "Givopel", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "logit_scale": 1.0,
                "logit_softcap": 50.0, "loop": {"start": 0, "stop": n, "times": 1}, "layers": [kinds[i % 2] for i in range(n)]}
    if design == "guzuvik":
        ssm = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 2, "conv": 4, "norm_groups": 2}
        attn = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 50.0, "v_mix": True,
                "mask": {"size": 1024, "keep_first": 4}}
        mlp = {"kind": "dense", "ff": inner}
        moe = {"kind": "moe", "expert": {"ff": inner // 8, "limit": 7.0}, "router": {"experts": 16, "top": 2}}
        kinds = [("mamba2", ssm, mlp), ("attention", attn, moe), ("mamba2", ssm, moe), ("attention", attn, mlp)]
        return {"architecture": "Guzuvik", "vocab": vocab, "width": width, "norm": {"eps": 1e-5},
                "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31337, "mul_cur": 7919}},
                "layers": [dict(zip(("type", "mixer", "mlp"), kinds[i % 4])) for i in range(n)]}
    rot = {"dims": dim // 2, "base": 500000.0}
    attn = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "rot": rot, "mask": {"size": 1024}}
    latent = {"heads": heads, "dim": dim, "rot_dim": 64, "vdim": dim, "kv_rank": 192, "scale": (dim + 64) ** -0.5,
              "rot": {"dims": 64, "base": 1000000.0}, "mask": {"size": 1024}}
    moe = {"kind": "moe", "expert": {"ff": inner // 8}, "router": {"experts": 16, "top": 2, "groups": {"count": 4, "keep": 2}}}
    layers = [{"type": "latent_attention", "mixer": latent, "mlp": moe} if i % 2 else
              {"type": "attention", "mixer": dict(attn, kv_from=i - 2) if i % 4 == 2 else attn, "mlp": moe} for i in range(n)]
    return {"architecture": "Zogevik", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "layers": layers}


def _spec(case):
    arch, config = xrt.config_from_dict(_config(case))
    return arch.build_spec(config)


def _draw_weights(case, seed):
    """{tensor name: tensor} as such models hold them: matrices of standard deviation 0.02, wide embeddings,
    and narrow what adds into the stream, the last matrices or the norms after them (a layer of a deep model changes the
    stream by a part of it), other norms around one, biases around zero, step sizes and decays of a state over tens to hundreds of tokens, routers whose
    choices stand out."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = {"bfloat16": torch.bfloat16, "float32": torch.float32}[case["dtype"]]

    def uniform(shape, low, high):
        return torch.rand(shape, generator=gen, device=DEVICE) * (high - low) + low

    weights = {}
    for e in _spec(case).expected_tensors():
        last = e.name.rsplit(".", 1)[-1]
        if e.kind == "matrix":
            wide = e.name in ("embed", "bigram", "model.embed_tokens.weight") and not case["model"].startswith("tiny")
            narrow = e.name.endswith(("o_proj.weight", "down_proj.weight"))
            std = 1.0 if wide else 0.0025 if narrow else 0.05 if last == "router" else 0.02
            t = torch.empty(e.shape, dtype=dtype, device=DEVICE).normal_(0.0, std, generator=gen)
        elif last == "A_log":
            t = uniform(e.shape, 1.0, 16.0).log()
        elif last == "dt_bias":
            t = uniform(e.shape, math.log(1e-3), math.log(1e-1)).exp().expm1().log()
        elif last == "conv":
            t = uniform(e.shape, -0.5, 0.5)
        elif last == "vmix":
            t = uniform(e.shape, 0.4, 0.6)
        elif last == "b":
            t = torch.empty(e.shape, device=DEVICE).normal_(2.0 if e.name.endswith("a2.b") else 0.0, 0.02, generator=gen)
        else:
            after = {"guzuvik": ("norm1b", "norm2b"), "zogevik": ("norm1", "norm2")}.get(case["model"].split("-")[0], ())
            t = torch.empty(e.shape, device=DEVICE).normal_(1.0, 0.1, generator=gen)
            t = t * 0.1 if last in after else t
        weights[e.name] = t
    return weights


def _lengths(case):
    rng = random.Random(case["batch"] * 7919 + case["longest"])
    return [rng.randint(case["shortest"], case["longest"]) for _ in range(case["batch"])]


def _tokens(case, vocab, seed):
    """(prompts, given ids of every step), uniform."""
    gen = torch.Generator().manual_seed(seed + 1)
    ids = lambda n: torch.randint(0, vocab, (n,), generator=gen).tolist()
    return [ids(n) for n in _lengths(case)], [ids(case["batch"]) for _ in range(case["steps"])]


# ----------------------------------------------------------------------------- the cases
def _model(name, model, layers, batch, shortest, longest, steps=0, scored=False, dtype="bfloat16", generate=False):
    case = {"kind": "model", "model": model, "layers": layers, "dtype": dtype, "batch": batch, "shortest": shortest,
            "longest": longest, "scored": scored, "steps": steps, "generate": generate}
    return dict(case, name=name) if name else case


def _sample(name, rows, vocab, temperature=0.8, top_k=40, top_p=0.95, penalty=1.1):
    case = {"kind": "sample", "rows": rows, "vocab": vocab, "temperature": temperature, "top_k": top_k, "top_p": top_p,
            "penalty": penalty}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest calls: a test-sized model in true 32-bit, greedy tokens from the sampler to the next step
        _model("tiny_f32_generate", "tiny-llama", 2, 3, 5, 13, steps=8, dtype="float32", generate=True),
        # the same in bfloat16, head norms and a tied output matrix: launches and host work are all there is
        _model("tiny_bf16_replay", "tiny-qwen3", 3, 4, 1, 31, steps=12),
        # time to the first token of one ordinary prompt at the size of an 8B model's layers
        _model("prompt_2048", "llama3-8b", 8, 1, 2048, 2048),
        # a long document: attention's share grows
        _model("prompt_7999", "llama3-8b", 8, 1, 7999, 7999),
        # a server's batch of prompts of very unequal lengths, with q/k norms
        _model("prompts_16_ragged", "qwen3-8b", 8, 16, 64, 2047),
        # a chat answer for one user
        _model("answer_b1", "llama3-8b", 8, 1, 500, 500, steps=60),
        # answers for a few users over a long context
        _model("answer_b8_long", "llama3-8b", 8, 8, 1500, 2048, steps=60),
        # answers for many users over short contexts
        _model("answer_b64", "qwen3-8b", 4, 64, 20, 300, steps=32),
        # the sampler with its default options over a large vocabulary, one row a user
        _sample("sample_64", 64, 128256),
        # layers with matrix states (gated linear attention, and a delta rule beside attention)
        _model("givopel_answer", "givopel-2k", 4, 1, 2000, 2000, steps=16),
        # state-space layers, capped attention in a window, routed experts; every token of the prompts is scored
        _model("guzuvik_score", "guzuvik-2k", 4, 2, 900, 1100, steps=8, scored=True),
        # latent attention and routed experts, a few users
        _model("zogevik_answer", "zogevik-2k", 4, 4, 100, 1500, steps=24, scored=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    what = rng.choice(["tiny", "prompt", "prompt", "answer", "answer", "answer", "design", "design", "design", "sample"])
    if what == "sample":
        return _sample(None, _log_int(rng, 1, 64), rng.choice([32000, 128256, 151936]), rng.choice([0.0, 0.7, 0.8, 1.0]),
                       rng.choice([0, 20, 40, 50]), rng.choice([0.9, 0.95, 1.0]), rng.choice([1.0, 1.1]))
    if what == "tiny":
        model = rng.choice(["tiny-llama", "tiny-qwen3"])
        dtype = rng.choice(["float32", "bfloat16"])
        longest = _log_int(rng, 4, 96)
        return _model(None, model, _DENSE[model][0], rng.randint(1, 8), rng.randint(1, longest), longest, rng.randint(1, 16),
                      rng.random() < 0.3, dtype, dtype == "float32" and rng.random() < 0.7)
    if what == "design":
        model = rng.choice(["givopel-2k", "guzuvik-2k", "zogevik-2k"])
        batch, scored, layers = _log_int(rng, 1, 16), not model.startswith("givopel"), 4
        tokens, steps = 4096, rng.randint(0, 24)
    else:
        model = rng.choice(["llama-2k", "llama3-8b", "qwen3-8b", "qwen3-32b"])
        layers = rng.randint(2, 8) if model != "qwen3-32b" else 2
        batch = _log_int(rng, 1, 16 if what == "prompt" else 64)
        tokens, steps, scored = 15000, 0 if what == "prompt" else rng.randint(8, 60), False
    longest = _log_int(rng, 20, min(tokens // batch, 8000))
    shortest = rng.choice([longest, max(1, longest // 16), rng.randint(1, longest)])
    return _model(None, model, layers, batch, shortest, longest, steps, scored)


# ----------------------------------------------------------------------------- one pass
def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    spec = _spec(case)
    dtype = xrt.parse_dtype(case["dtype"])
    model = xrt.Model(spec, _draw_weights(case, seed), dtype, DEVICE)
    prompts, given = _tokens(case, spec.vocab_size, seed)
    held = sum(-(-(len(p) + case["steps"]) // BLOCK_TOKENS) * BLOCK_TOKENS for p in prompts)
    engine = xrt.Engine(model, held, max_slots=len(prompts))
    state = {"engine": engine, "prompts": prompts, "steps": [[[t] for t in row] for row in given], "scored": case["scored"]}
    if case["generate"]:
        state["sampler"] = Sampler(engine.cache, spec.vocab_size)
        state["options"] = [SamplerConfig(0.0, 0, 1.0, 1.0)] * len(prompts)
    return state


def run(state):
    if "logits" in state:
        return {"ids": state["sampler"].sample(state["logits"], state["rows"], state["options"])}
    engine, prompts = state["engine"], state["prompts"]
    slots = [engine.open_slot() for _ in prompts]
    want = lambda p: list(range(len(p))) if state["scored"] else [len(p) - 1]
    logits = engine.step([xrt.StepEntry(s, p, want(p)) for s, p in zip(slots, prompts)])
    out, rows = {"prompt": logits}, []
    if "sampler" in state:
        sampler, chosen = state["sampler"], []
        sampler.begin(slots, list(range(len(slots))))
        row_slot = engine.last_context.seq_slot[:len(slots)]
        for i in range(len(state["steps"])):
            chosen.append(sampler.sample(logits, row_slot, state["options"]))
            logits = engine.step_sampled(slots, chosen[-1])
            row_slot = engine.last_context.seq_slot[:len(slots)]
            rows.append(logits)
        out["ids"] = torch.stack(chosen)
    else:
        for given in state["steps"]:
            rows.append(engine.step([xrt.StepEntry(s, t, [0]) for s, t in zip(slots, given)]))
    if rows:
        out["steps"] = torch.stack(rows)
    for s in slots:
        engine.close_slot(s)
    return out


def _prepare_sample(case, seed):
    """Logits as an output matrix gives them, and sequences that have seen some hundred ids."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    rows, vocab = case["rows"], case["vocab"]
    cache = Cache([], rows * BLOCK_TOKENS, 16384, xrt.DType.BF16, DEVICE, rows)
    sampler = Sampler(cache, vocab)
    slots = [cache.open_slot() for _ in range(rows)]
    sampler.begin(slots, [seed + i for i in range(rows)])
    row_slot = torch.tensor(slots, dtype=torch.int32, device=DEVICE)
    seen = torch.randint(0, vocab, (rows * 200,), generator=gen, device=DEVICE, dtype=torch.int32)
    sampler.observe(row_slot.repeat_interleave(200), seen)
    logits = torch.empty((rows, vocab), device=DEVICE).normal_(0.0, 3.0, generator=gen)
    options = [SamplerConfig(case["temperature"], case["top_k"], case["top_p"], case["penalty"])] * rows
    return {"sampler": sampler, "logits": logits, "rows": row_slot, "options": options}


# ----------------------------------------------------------------------------- what a pass cannot do without
def _mixer_work(layer, width, lengths):
    """(bytes of keys, values and state, operations) of one layer's mixer over sequences of ``lengths`` [(before, new)],
    without its matrices."""
    kind, m = layer["type"], layer["mixer"]
    byte = flop = 0.0
    parts = [("attention", m["left"]), ("scan", m["right"])] if kind == "parallel" else \
        [("attention" if kind in ("attention", "latent_attention") else "scan", m)]
    for part, p in parts:
        for before, new in lengths:
            if part == "scan":
                size = p["heads"] * p["vdim"] * p.get("dim", p.get("state", 0))
                byte += 8.0 * size
                flop += 4.0 * size * new  # the update and the read-out
                continue
            seen = float(sum(min((p.get("mask") or {}).get("size") or before + i + 1, before + i + 1) for i in range(new)))
            latent = kind == "latent_attention"
            row = p["kv_rank"] + p["rot_dim"] if latent else p["kv_heads"] * (p["dim"] + p["vdim"])
            qk, pv = (p["dim"] + p["rot_dim"], p["vdim"]) if latent else (p["dim"], p["vdim"])
            byte += 2.0 * row * (min(before + new, (p.get("mask") or {}).get("size") or before + new) + new)
            flop += 2.0 * p["heads"] * (qk + pv) * seen
    return byte, flop


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 0.0}
    config = _config(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    if "hidden_size" in config:
        c = config
        width, vocab = c["hidden_size"], c["vocab_size"]
        mixer = {"heads": c["num_attention_heads"], "kv_heads": c["num_key_value_heads"], "dim": c["head_dim"],
                 "vdim": c["head_dim"]}
        layers = [{"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": c["intermediate_size"]}}] * case["layers"]
    else:
        width, vocab, layers = config["width"], config["vocab"], config["layers"]
    head = embed = expert = other = 0
    routed = []
    for e in _spec(case).expected_tensors():
        if e.kind != "matrix":
            continue
        count = math.prod(e.shape)
        parts = e.name.split(".")
        if e.name in ("lm_head.weight", "head"):
            head = count
        elif e.name in ("embed", "bigram", "model.embed_tokens.weight"):
            embed = count if e.name != "bigram" else embed
        elif len(parts) == 4 and parts[1] == "mlp" and parts[2][0] == "e" and parts[2][1:].isdigit():
            expert += count
        else:
            other += count
    head = head or embed
    for layer in layers:
        mlp = layer.get("mlp") or {}
        if mlp.get("kind") == "moe":
            routed.append(mlp["router"])
    lengths, byte, flop = _lengths(case), 0.0, 0.0
    for step in range(case["steps"] + 1):
        spans = [(0, n) if step == 0 else (n + step - 1, 1) for n in lengths]
        tokens = sum(new for _, new in spans)
        rows = tokens if step == 0 and case["scored"] else len(spans)
        share = 1.0  # of the experts' matrices that a step reads, and a token's share of their operations
        if routed:
            n, top = routed[0]["experts"], routed[0]["top"]
            share = 1.0 - (1.0 - top / n) ** tokens
            flop += 2.0 * expert * top / n * tokens
        byte += size * (other + head + share * expert + tokens * width) + 4.0 * rows * vocab
        flop += 2.0 * other * tokens + 2.0 * head * rows
        for layer in layers:
            b, f = _mixer_work(layer, width, spans)
            byte += b * (size / 2 if layer["type"] == "attention" else 1)
            flop += f
    return {"bytes": byte, "flops": flop}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.0}
    # routed experts: a token whose router's choice is a near tie takes another expert, and its row moves with it
    return {"rel": 0.03, "max": 0.99} if case["model"].split("-")[0] in ("guzuvik", "zogevik") else {"rel": 0.03, "max": 0.3}


# ----------------------------------------------------------------------------- 64-bit restatement
F64 = torch.float64


def _rms(x, w=None, eps=0.0):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _layer_norm(x, w, b, eps):
    d = x - x.mean(-1, keepdim=True)
    y = d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w
    return y if b is None else y + b


def _rotate(x, freqs, interleaved, mult=1.0):
    """x [T, heads, dim] of one sequence from position 0; the first 2 * len(freqs) dims of every head turn."""
    n = 2 * freqs.numel()
    angle = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * freqs[None, :]
    cos, sin = angle.cos()[:, None] * mult, angle.sin()[:, None] * mult
    first, second = (slice(0, n, 2), slice(1, n, 2)) if interleaved else (slice(0, n // 2), slice(n // 2, n))
    out = x.clone()
    out[..., first] = x[..., first] * cos - x[..., second] * sin
    out[..., second] = x[..., second] * cos + x[..., first] * sin
    return out


def _frequencies(dims, base, scaling=None):
    i = torch.arange(dims // 2, dtype=F64, device=DEVICE)
    f = torch.tensor(base, dtype=F64, device=DEVICE) ** (-2.0 * i / dims)
    if not scaling:
        return f, 1.0
    dim_of = lambda turns: dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(dim_of(scaling["fast"])), 0), min(math.ceil(dim_of(scaling["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / scaling["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0


def _attend(q, k, v, scale, window=None, keep_first=0, cap=None, slopes=None, sink=False):
    """Causal grouped-query attention of one sequence: q [T, H, d], k [T, G, d], v [T, G, e] -> [T, H * e]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    at = torch.arange(T, device=q.device)
    back = at[:, None] - at[None, :]
    hidden = back < 0
    if window:
        hidden = hidden | ((back >= window) & (at[None, :] >= keep_first))
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h] * back
        s = s.masked_fill(hidden, -math.inf)
        m = s.max(-1, keepdim=True).values
        m = m.clamp(min=0.0) if sink else m
        p = torch.exp(s - m)
        out[:, h] = (p / (p.sum(-1, keepdim=True) + (torch.exp(-m) if sink else 0.0))) @ v[:, h // (H // G)]
    return out.reshape(T, -1)


def _scan(q, k, v, decay, beta, lengths):
    """S <- decay * S (rows); u = v, or beta (v - S^T k); S <- S + k u^T; o = S^T q, token by token for all sequences and
    heads at once.  Flat rows [sum T, H, dim], beta [sum T, H] or None; decay may be one number a head."""
    pad = lambda x: torch.nn.utils.rnn.pad_sequence(list(x.split(lengths)), batch_first=True)
    q, k, v, decay = pad(q), pad(k), pad(v), pad(decay.expand(-1, -1, k.shape[2]))
    beta = pad(beta) if beta is not None else None
    S = torch.zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3], dtype=F64, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[1]):
        S = S * decay[:, t].unsqueeze(-1)
        u = v[:, t]
        if beta is not None:
            u = beta[:, t].unsqueeze(-1) * (u - (k[:, t].unsqueeze(-2) @ S).squeeze(-2))
        S = S + k[:, t].unsqueeze(-1) * u.unsqueeze(-2)
        out[:, t] = (q[:, t].unsqueeze(-2) @ S).squeeze(-2)
    return torch.cat([row[:n] for row, n in zip(out, lengths)])


def _conv(x, taps, bias, lengths):
    out = []
    for row in x.split(lengths):
        padded = torch.cat([row.new_zeros(taps.shape[1] - 1, row.shape[1]), row])
        out.append(sum(padded[j:j + row.shape[0]] * taps[:, j] for j in range(taps.shape[1])))
    y = torch.cat(out)
    return y if bias is None else y + bias


def _each(lengths, f, *flat):
    return torch.cat([f(*rows) for rows in zip(*(x.split(lengths) for x in flat))])


_silu = torch.nn.functional.silu
_softplus = torch.nn.functional.softplus


def _dense_layers(w, c, x, lengths):
    H, G, d, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
    freqs, _ = _frequencies(d, c["rope_theta"])
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w(p + "input_layernorm.weight"), eps)
        q, k, v = ((h @ w(p + f"self_attn.{r}_proj.weight").T).view(len(h), -1, d) for r in "qkv")
        if c["architectures"][0] == _QWEN3:
            q, k = _rms(q, w(p + "self_attn.q_norm.weight"), eps), _rms(k, w(p + "self_attn.k_norm.weight"), eps)
        att = _each(lengths, lambda q, k, v: _attend(_rotate(q, freqs, False), _rotate(k, freqs, False), v, d ** -0.5), q, k, v)
        x = x + att @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, w(p + "post_attention_layernorm.weight"), eps)
        up = _silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)
        x = x + up @ w(p + "mlp.down_proj.weight").T
    return _rms(x, w("model.norm.weight"), eps)


def _givopel_layers(w, c, x, lengths):
    eps, x0 = c["norm"]["eps"], x
    x = torch.cat([x, x0], -1) @ w("loop.in").T  # the only pass of the loop begins with the first layer
    for i, layer in enumerate(c["layers"]):
        h = _layer_norm(x, w(f"l{i}.norm1"), None, eps)
        p, m = f"l{i}.mix.", layer["mixer"]
        heads = lambda t, n: t.view(len(t), n, -1)
        lin = lambda name, y=h: y @ w(p + name).T
        if layer["type"] == "gla":
            n = m["heads"]
            decay = torch.sigmoid(lin("a2", lin("a1")) + w(p + "a2.b")) ** (1.0 / m["tau"])
            o = _scan(heads(lin("q"), n) * m["dim"] ** -0.5, heads(lin("k"), n), heads(lin("v"), n), heads(decay, n), None, lengths)
            y = lin("o", _rms(o, w(p + "norm"), eps).flatten(1) * _silu(lin("g")))
        else:
            a, b = m["left"], m["right"]
            freqs, mult = _frequencies(a["rot"]["dims"], a["rot"]["base"], a["rot"]["scaling"])
            turn = lambda t: _rotate(t, freqs, True, mult)
            att = _each(lengths, lambda q, k, v: _attend(turn(q), turn(k), v, a["scale"]), heads(lin("left.q"), a["heads"]),
                        heads(lin("left.k"), a["kv_heads"]), heads(lin("left.v"), a["kv_heads"]))
            left = lin("left.o", att * torch.sigmoid(lin("left.g")))
            n, per = b["heads"], b["heads"] // b["kv_heads"]
            q, k, v = (_silu(_conv(lin("right." + r), w(p + f"right.{r}.conv"), None, lengths)) for r in "qkv")
            unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
            q = (unit(heads(q, b["kv_heads"])) * b["dim"] ** -0.5).repeat_interleave(per, 1)
            k = unit(heads(k, b["kv_heads"])).repeat_interleave(per, 1)
            step = heads(_softplus(lin("right.a2", lin("right.a1")) + w(p + "right.dt_bias")), n)
            decay = torch.exp(-torch.exp(w(p + "right.A_log"))[None, :, None] * step)
            o = _scan(q, k, heads(v, n), decay, torch.sigmoid(lin("right.b")), lengths)
            gate = torch.sigmoid(lin("right.g2", lin("right.g1")))
            right = lin("right.o", _rms(o, w(p + "right.norm"), eps).flatten(1) * gate)
            y = 0.5 * (_rms(left, w(p + "left.out"), eps) + _rms(right, w(p + "right.out"), eps))
        p = f"l{i}.mlp."
        x = x + y + lin("down", _silu(lin("gate")) * lin("up"))
    return _layer_norm(x, w("final.norm"), None, eps)


def _experts(w, p, h, chosen, weights, unit):
    out = torch.zeros_like(h)
    for e in range(int(chosen.max()) + 1):
        token, which = (chosen == e).nonzero(as_tuple=True)
        if token.numel():
            out.index_add_(0, token, weights[token, which, None] * (unit(h[token], f"{p}e{e}.") @ w(f"{p}e{e}.down").T))
    return out


def _guzuvik_layers(w, c, x, lengths):
    eps, v_first = c["norm"]["eps"], None
    for i, layer in enumerate(c["layers"]):
        norm = lambda name, y: _layer_norm(y, w(f"l{i}.{name}"), w(f"l{i}.{name}.b"), eps)
        h, p, m = norm("norm1", x), f"l{i}.mix.", layer["mixer"]
        n = m["heads"]
        if layer["type"] == "mamba2":
            inner, gn = n * m["vdim"], m["groups"] * m["state"]
            z, xbc, dt = (h @ w(p + "in").T).split([inner, inner + 2 * gn, n], -1)
            u, b, k = _silu(_conv(xbc, w(p + "conv"), w(p + "conv.b"), lengths)).split([inner, gn, gn], -1)
            dt = _softplus(dt + w(p + "dt_bias"))
            wide = lambda t: t.view(len(t), m["groups"], -1).repeat_interleave(n // m["groups"], 1)
            u = u.view(len(u), n, -1)
            y = _scan(wide(k), wide(b) * dt[..., None], u, torch.exp(-torch.exp(w(p + "A_log")) * dt)[..., None], None, lengths)
            y = (y + w(p + "D")[:, None] * u).flatten(1) * _silu(z)
            y = _rms(y.view(len(y), m["norm_groups"], -1), None, eps).flatten(1) * w(p + "norm")
        else:
            q, k, v = ((h @ w(p + r).T + w(p + r + ".b")).view(len(h), -1, m["dim"]) for r in "qkv")
            v_first = v if v_first is None else v_first
            lam = w(p + "vmix")
            v = v if v is v_first else (1.0 - lam) * v + lam * v_first
            slopes = [2.0 ** (-8.0 * (a + 1) / n) for a in range(n)]
            y = _each(lengths, lambda q, k, v: _attend(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"],
                                                       m["softcap"], slopes), _rms(q, None, eps), _rms(k, None, eps), v)
            y = (y.view(len(y), n, -1) * torch.sigmoid(h @ w(p + "g").T)[..., None]).flatten(1)
        x = x + norm("norm1b", y @ w(p + "o").T)
        h, p, mlp = norm("norm2", x), f"l{i}.mlp.", layer["mlp"]
        if mlp["kind"] == "dense":
            y = torch.relu(h @ w(p + "up").T) ** 2 @ w(p + "down").T
        else:
            limit = mlp["expert"]["limit"]

            def unit(t, e):
                g, u = (t @ w(e + "gate").T).clamp(max=limit), (t @ w(e + "up").T).clamp(-limit, limit)
                return g * torch.sigmoid(1.702 * g) * (u + 1.0)

            best, chosen = (h @ w(p + "router").T + w(p + "router.b")).topk(mlp["router"]["top"], -1)
            y = _experts(w, p, h, chosen, best.softmax(-1), unit)
        x = x + norm("norm2b", y)
    return _layer_norm(x, w("final.norm"), w("final.norm.b"), eps)


def _zogevik_layers(w, c, x, lengths):
    eps, kept = c["norm"]["eps"], {}
    x = _rms(x, w("embed.norm"), eps)
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        n, window = m["heads"], m["mask"]["size"]
        freqs, _ = _frequencies(m["rot"]["dims"], m["rot"]["base"])
        if layer["type"] == "attention":
            turn = lambda t: _each(lengths, lambda s: _rotate(s, freqs, False), t.view(len(t), -1, m["dim"]))
            if "kv_from" not in m:
                kept[i] = (turn(_rms(x @ w(p + "k").T, w(p + "k.norm"), eps)), (x @ w(p + "v").T).view(len(x), -1, m["vdim"]))
            k, v = kept[m.get("kv_from", i)]
            q = turn(_rms(x @ w(p + "q").T, w(p + "q.norm"), eps))
            y = _each(lengths, lambda q, k, v: _attend(q, k, v, m["scale"], window, sink=True), q, k, v)
        else:
            turn = lambda t: _each(lengths, lambda s: _rotate(s, freqs, True), t)
            q = (x @ w(p + "q").T).view(len(x), n, -1)
            down = x @ w(p + "dkv").T
            latent = _rms(down[:, :m["kv_rank"]], w(p + "dkv.norm"), eps)
            shared = turn(down[:, None, m["kv_rank"]:]).expand(-1, n, -1)
            q = torch.cat([q[..., :m["dim"]], turn(q[..., m["dim"]:])], -1)
            k = torch.cat([(latent @ w(p + "uk").T).view(len(x), n, -1), shared], -1)
            v = (latent @ w(p + "uv").T).view(len(x), n, -1)
            y = _each(lengths, lambda q, k, v: _attend(q, k, v, m["scale"], window), q, k, v)
        x = x + _rms(y @ w(p + "o").T, w(f"l{i}.norm1"), eps)
        p, r = f"l{i}.mlp.", layer["mlp"]["router"]
        scores = (x @ w(p + "router").T).softmax(-1)
        grouped = scores.view(len(x), r["groups"]["count"], -1)
        keep = grouped.max(-1).values.topk(r["groups"]["keep"], -1).indices
        allowed = torch.zeros(grouped.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, keep, True)
        best, chosen = grouped.masked_fill(~allowed[..., None], -1.0).flatten(1).topk(r["top"], -1)
        unit = lambda t, e: torch.nn.functional.gelu(t @ w(e + "up").T)
        x = x + _rms(_experts(w, p, x, chosen, best, unit), w(f"l{i}.norm2"), eps)
    return _rms(x, w("final.norm"), eps)


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    config = _config(case)
    weights = _draw_weights(case, seed)
    w = lambda name: weights[name].to(F64)
    vocab = config.get("vocab_size") or config["vocab"]
    prompts, given = _tokens(case, vocab, seed)
    steps = case["steps"]
    if case["generate"]:  # the ids follow from the logits: the plain model goes on from its own, step by step
        rows = [list(p) for p in prompts]
        out = _forward(case, config, w, rows)
        first, more = [r[-1] for r in out], []
        if case["scored"]:
            scored = torch.cat(out)
        latest = first
        for _ in range(steps):
            rows = [r + [int(l.argmax())] for r, l in zip(rows, latest)]
            latest = [r[-1] for r in _forward(case, config, w, rows)]
            more.append(torch.stack(latest))
        answer = {"ids": None, "prompt": scored if case["scored"] else torch.stack(first)}
        return dict(answer, steps=torch.stack(more)) if steps else answer
    rows = [p + [row[b] for row in given] for b, p in enumerate(prompts)]
    # only the wanted rows pass the output matrix: a prompt's last (or every) token, and the steps' tokens
    out = _forward(case, config, w, rows, [0 if case["scored"] else len(p) - 1 for p in prompts])
    cut = [r.shape[0] - steps for r in out]
    answer = {"prompt": torch.cat([r[:n] for r, n in zip(out, cut)])}
    if steps:
        answer["steps"] = torch.stack([r[n:] for r, n in zip(out, cut)], 1)
    return answer


def _forward(case, config, w, rows, first=None):
    """Logits of every sequence's tokens from place ``first[i]`` on."""
    lengths = [len(r) for r in rows]
    ids = torch.tensor([t for r in rows for t in r], device=DEVICE)
    embed = "model.embed_tokens.weight" if "hidden_size" in config else "embed"
    x = w(embed)[ids]
    design = case["model"].split("-")[0]
    if design == "guzuvik":
        pair, pairs = config["embedding"]["bigram"], []
        for r in rows:
            pairs += [pair["buckets"]] + [(a * pair["mul_prev"] + b * pair["mul_cur"]) % pair["buckets"] for a, b in zip(r, r[1:])]
        x = x + w("bigram")[torch.tensor(pairs, device=DEVICE)]
    layers = {"givopel": _givopel_layers, "guzuvik": _guzuvik_layers, "zogevik": _zogevik_layers}.get(design, _dense_layers)
    x = layers(w, config, x, lengths)
    x = torch.cat([s[a:] for s, a in zip(x.split(lengths), first or [0] * len(lengths))])
    if "hidden_size" in config:
        head = embed if config["tie_word_embeddings"] else "lm_head.weight"
    else:
        head = "embed" if design == "guzuvik" else "head"
    logits = x @ w(head).T
    if config.get("logit_softcap"):
        logits = config["logit_softcap"] * torch.tanh(logits * config["logit_scale"] / config["logit_softcap"])
    return list(logits.split([n - a for n, a in zip(lengths, first or [0] * len(lengths))]))
