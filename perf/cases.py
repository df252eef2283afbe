"""The work this engine is measured on: whole waves of requests through the step function, and the sampler.

A wave is what a service sees: requests arrive together, prompts are cut into portions under a budget of 2,048 tokens a
step (running requests decode first, the rest of the budget goes to prompts in arrival order, so that most waves hold
prompt portions beside decoded tokens), every request decodes its tokens, then all are finished.  The tokens are given
(as in a trace replay or a perplexity run), so the outputs are the logits at every place a token is drawn from.

Models have the layer widths of this repository's benchmark and of its tests at real widths, with fewer layers (four, or
one turn of a design's own pattern of layers) so that a state is made in well under a second; every kernel of a layer runs
at its full size, and the LM head weighs more than in the whole model.  Weights are random (matrices N(0, 0.02) and so on,
as the random-weights mode draws them; decays and time steps of the state-space mixers as they are commonly initialised).

`listed()` names what each case stands for.  `draw()` spreads over the models, 1 to 64 requests, prompts of 8 to 8,191 tokens,
1 to 64 new tokens, both types; and over 1 to 64 rows of three vocabularies for the sampler.
"""
import math
import random
import zlib

import numpy as np
import torch

from rvllm_b200 import Engine, EngineConfig, Sampler, SamplingParams, StepEntry, config_from_dict
from rvllm_b200.kernels import get_library
from rvllm_b200.models.decoder import expected_tensors

DEVICE = "cuda:0"
BUDGET = 2048                    # tokens a step, the engine's default
GRAPH_SIZES = (1, 2, 4, 8, 16, 32, 64)
VOCAB = 32768                    # of the designs whose benchmark workloads use it
F64 = torch.float64


# ------------------------------------------------------------------------------------------------------------- models
def _dense(arch, hidden, layers, heads, kv, dim, ff, vocab, theta, eps, tie, scaling=None):
    cfg = {"architectures": [arch], "hidden_size": hidden, "num_hidden_layers": layers, "num_attention_heads": heads,
           "num_key_value_heads": kv, "head_dim": dim, "intermediate_size": ff, "vocab_size": vocab, "max_position_embeddings": 32768,
           "rms_norm_eps": eps, "rope_theta": theta, "tie_word_embeddings": tie, "hidden_act": "silu", "torch_dtype": "bfloat16"}
    if scaling:
        cfg["rope_scaling"] = scaling
    return cfg


def _tufirax(width, heads, kv, rot, ff, m_heads):
    """Attention with whole-row q/k norms, a sink and a gate, and mamba2, in turn."""
    att = {"type": "attention", "mixer": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
                                          "rot": {"dims": rot, "base": 500000.0}}, "mlp": {"kind": "dense", "ff": ff}}
    mam = {"type": "mamba2", "mixer": {"heads": m_heads, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8},
           "mlp": {"kind": "dense", "ff": ff}}
    return {"architecture": "Tufirax", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-6}, "layers": [att, mam] * 2}


def _latent(heads):
    return {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 192, "scale": 192 ** -0.5,
            "rot": {"dims": 64, "base": 500000.0}}


def _vipelix(width, heads, ff, e_ff, experts, top, shared):
    """Latent attention; a dense layer and a layer of table-routed experts, both run twice."""
    moe = {"kind": "moe", "expert": {"ff": e_ff}, "router": {"experts": experts, "top": top}, "shared": {"ff": shared}}
    layers = [{"type": "latent_attention", "mixer": _latent(heads), "mlp": m} for m in ({"kind": "dense", "ff": ff}, moe)]
    return {"architecture": "Vipelix", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "loop": {"start": 0, "stop": 2, "times": 2}, "layers": layers}


def _tibepel(width, heads, kv, ff, r_heads, r_kv, inner, rank):
    """Attention with mixed head weights beside a gated delta rule, and mamba1, in turn."""
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    par = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 4096}}, "left_scale": 0.7,
        "right": {"heads": r_heads, "kv_heads": r_kv, "dim": 128, "vdim": 128, "conv": 4}, "right_scale": 0.7}}
    mam = {"type": "mamba1", "mlp": mlp, "mixer": {"inner": inner, "state": 16, "dt_rank": rank, "conv": 4}}
    return {"architecture": "Tibepel", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0},
            "logit_softcap": 30.0, "token_side": {"dim": 64}, "layers": [par, mam] * 2}


def _tugodra(width, heads, kv, m_heads, e_ff, experts, top, groups, keep, shared):
    """A matrix memory, window attention on unit vectors, latent attention with a sink, window attention on borrowed keys."""
    mlp = {"kind": "moe", "expert": {"ff": e_ff}, "shared": {"ff": shared},
           "router": {"experts": experts, "top": top, "groups": {"count": groups, "keep": keep}}}
    att = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** 0.5 * 0.1, "mask": {"size": 1024},
           "rot": {"dims": 128, "base": 1e6}}
    mixers = [("mlstm", {"heads": m_heads, "dim": 128, "vdim": 256, "gate_cap": 15.0}), ("attention", att),
              ("latent_attention", _latent(heads)), ("attention", dict(att, kv_from=1))]
    return {"architecture": "Tugodra", "width": width, "vocab": VOCAB, "norm": {"eps": 1e-6}, "embedding": {"scale": width ** 0.5},
            "layers": [{"type": t, "mixer": m, "mlp": mlp} for t, m in mixers]}


LLAMA3 = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}
MODELS = {
    "llama-8b": lambda: _dense("LlamaForCausalLM", 4096, 4, 32, 8, 128, 14336, 128256, 500000.0, 1e-5, False, LLAMA3),
    "qwen-7b": lambda: _dense("Qwen2ForCausalLM", 3584, 4, 28, 4, 128, 18944, 152064, 1000000.0, 1e-6, False),
    "qwen-0.5b": lambda: _dense("Qwen2ForCausalLM", 896, 4, 14, 2, 64, 4864, 151936, 1000000.0, 1e-6, True),
    "tufirax-2k": lambda: _tufirax(2048, 16, 4, 64, 8192, 64),
    "tufirax-4k": lambda: _tufirax(4096, 32, 8, 128, 14336, 128),
    "vipelix-2k": lambda: _vipelix(2048, 16, 8192, 1408, 16, 2, 2816),
    "vipelix-4k": lambda: _vipelix(4096, 32, 14336, 2048, 32, 4, 4096),
    "tibepel-2k": lambda: _tibepel(2048, 16, 4, 8192, 16, 8, 4096, 128),
    "tibepel-4k": lambda: _tibepel(4096, 32, 8, 14336, 32, 16, 8192, 256),
    "tugodra-2k": lambda: _tugodra(2048, 16, 4, 8, 1408, 16, 2, 4, 2, 2816),
    "tugodra-4k": lambda: _tugodra(4096, 32, 8, 16, 2048, 32, 4, 8, 4, 4096),
}
DENSE = ("llama-8b", "qwen-7b", "qwen-0.5b")


# -------------------------------------------------------------------------------------------------------------- cases
def _wave(name, model, requests, shortest, longest, new, dtype="bfloat16"):
    return {"name": name, "kind": "wave", "model": model, "dtype": dtype, "requests": requests, "shortest": shortest,
            "longest": longest, "new": new}


def listed():
    return [
        # a short question to a small model: latency and launches
        _wave("qwen-0.5b one question", "qwen-0.5b", 1, 17, 17, 16),
        # one user's chat turn on the model of the default benchmark: decode of one sequence
        _wave("llama-8b one request", "llama-8b", 1, 203, 203, 64),
        # the default benchmark: eight 2,048-token prompts, then decode of eight sequences
        _wave("llama-8b eight requests", "llama-8b", 8, 2048, 2048, 64),
        # a full batch of uneven chats: decode of 64 sequences, prompt portions beside them
        _wave("qwen-7b full batch", "qwen-7b", 64, 33, 517, 32),
        # a document: one long prompt in portions, a few tokens of answer
        _wave("llama-8b long prompt", "llama-8b", 1, 8191, 8191, 4),
        # the 32-bit path, in which correctness is judged
        _wave("qwen-7b float32", "qwen-7b", 3, 57, 190, 8, "float32"),
        # the other designs at the sizes of their benchmark workloads: prompts of an article's length, then decode
        _wave("tufirax-4k four requests", "tufirax-4k", 4, 300, 1500, 32),
        _wave("vipelix-4k eight requests", "vipelix-4k", 8, 150, 900, 32),
        _wave("tibepel-4k four requests", "tibepel-4k", 4, 300, 1500, 32),
        _wave("tugodra-4k four requests", "tugodra-4k", 4, 300, 1500, 32),
        # one long prompt on the smaller size of a design
        _wave("tibepel-2k one prompt", "tibepel-2k", 1, 3001, 3001, 8),
        # the draw of a batch's next tokens, every request with parameters of its own
        {"name": "sample 64 rows", "kind": "sample", "rows": 64, "vocab": 128256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.1:
        return {"kind": "sample", "rows": _log(rng, 1, 64), "vocab": rng.choice([32768, 128256, 152064])}
    model = rng.choice(["llama-8b", "qwen-7b"]) if rng.random() < 0.4 else rng.choice(sorted(MODELS))
    dtype = "float32" if model in DENSE and rng.random() < 0.15 else "bfloat16"
    # tokens of all prompts, and logits rows: no more than the largest listed case
    most = 600 if dtype == "float32" else 16384 if model in DENSE else 4096
    requests = _log(rng, 1, 8 if dtype == "float32" else 64)
    longest = min(_log(rng, 8, 8191), most // requests)
    shortest = rng.randint(max(1, longest // 8), longest)
    new = min(_log(rng, 1, 8 if dtype == "float32" else 64 if model in DENSE else 32), max(1, 2048 // requests))
    c = _wave("", model, requests, shortest, longest, new, dtype)
    del c["name"]
    return c


def lengths(case):
    """The prompts' lengths, spread evenly over the range in a mixed order; the same for every seed."""
    lo, hi = case["shortest"], case["longest"]
    return [lo + int((hi - lo + 1) * ((i * 0.6180339887498949 + 0.37) % 1.0)) for i in range(case["requests"])]


def plan(case):
    """The wave's steps: lists of (request, first position, number of tokens, whether its last place's logits are wanted)."""
    prompt, new = lengths(case), case["new"]
    done, steps = [0] * len(prompt), []
    total = [n + new - 1 for n in prompt]                       # the last token drawn is not fed back
    while any(d < t for d, t in zip(done, total)):
        step, room = [], BUDGET
        for r, n in enumerate(prompt):
            if n <= done[r] < total[r]:
                step.append((r, done[r], 1, True))
                room -= 1
        for r, n in enumerate(prompt):
            if done[r] < n and room > 0:
                k = min(room, n - done[r])
                step.append((r, done[r], k, done[r] + k == n))
                room -= k
        for r, _, k, _ in step:
            done[r] += k
        steps.append(step)
    return steps


def token_ids(case, seed, vocab):
    rng = np.random.default_rng([int(seed), 11])
    return [rng.integers(0, vocab, n + case["new"] - 1).tolist() for n in lengths(case)]


# ------------------------------------------------------------------------------------------------------------ weights
_INIT = {"matrix": (0.0, 0.02), "norm": (1.0, 0.1), "bias": (0.0, 0.02), "conv_taps": (0.0, 0.3), "coef": (0.5, 0.3),
         "mixing": (0.0, 0.3), "unit_scale": (0.7, 0.1)}


def tensor(seed, name, shape, init, dtype):
    """One weight on the device, from the seed and its name alone."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed((int(seed) << 32) + zlib.crc32(name.encode()))
    if init.startswith("choice:"):
        scores = torch.rand((shape[0], int(init[7:])), generator=gen, device=DEVICE)
        return scores.topk(shape[1], dim=1).indices.to(torch.int32).contiguous()
    t = torch.empty(shape, dtype=torch.float32, device=DEVICE)
    if name.endswith("A_log"):                                   # decay rates between 1 and 16
        t = t.uniform_(1.0, 16.0, generator=gen).log_()
    elif name.endswith("dt_bias") or name.endswith("dt.b"):      # time steps between 0.001 and 0.1
        dt = t.uniform_(math.log(1e-3), math.log(1e-1), generator=gen).exp_()
        t = dt + torch.log(-torch.expm1(-dt))
    elif name.endswith("mix.f.b"):                               # forget gates that keep most
        t = t.uniform_(3.0, 6.0, generator=gen)
    else:
        mean, std = _INIT[init]
        if ".mlp.e" in name and name.endswith(".down"):          # experts share a layer's output: one expert more or less is a small part of it
            std *= 0.5
        t = t.normal_(mean, std, generator=gen)
        if name.endswith(".r1") or name.endswith(".r2"):
            t = t.abs_()
    return t.to(dtype)


# ------------------------------------------------------------------------------------------------------ what is timed
def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    cfg = MODELS[case["model"]]()
    config = config_from_dict(cfg)
    prompt, n_req = lengths(case), case["requests"]
    longest = max(prompt) + case["new"]
    pages = sum((n + case["new"] + 15) // 16 + 1 for n in prompt) + 8
    engine = Engine(config=config, random_weights=True, seed=int(seed), engine_config=EngineConfig(
        dtype=case["dtype"], num_blocks=pages, max_model_len=(longest + 15) // 16 * 16, max_num_seqs=n_req, max_num_batched_tokens=max(BUDGET, n_req),
        cuda_graph_batch_sizes=GRAPH_SIZES, device=DEVICE))
    specs = engine.model.expected_tensors()
    engine.model.load(lambda name: tensor(seed, name, specs[name].shape, specs[name].init, engine.dtype), engine.dtype, engine.device,
                      engine.config.max_model_len)
    ids = token_ids(case, seed, config.vocab_size)
    steps = [[StepEntry(r, ids[r][a:a + k], (k - 1,) if want else ()) for r, a, k, want in step] for step in plan(case)]
    # the decode graphs are captured before the first request, as a service does when it starts
    decodes = {len(s) for s in steps if all(len(e.tokens) == 1 and len(e.want) == 1 for e in s)}
    sizes = sorted({min(b for b in GRAPH_SIZES if b >= n) for n in decodes})
    if sizes:
        engine.runner.capture_decode_graphs(longest, sizes)
    return {"runner": engine.runner, "steps": steps, "requests": range(n_req), "rows": n_req * case["new"], "vocab": config.vocab_size}


def _prepare_sample(case, seed):
    R, V = case["rows"], case["vocab"]
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(int(seed))
    # most of a vocabulary is noise, a few dozen tokens stand out
    logits = torch.randn((R, V), generator=gen, device=DEVICE) * 1.6
    likely = torch.randint(0, V, (R, 40), generator=gen, device=DEVICE)
    logits.scatter_add_(1, likely, torch.rand((R, 40), generator=gen, device=DEVICE) * 9.0 + 2.0)
    kinds = [SamplingParams(temperature=0.8, top_k=50, top_p=0.95), SamplingParams(temperature=0.7, top_p=0.9), SamplingParams(),
             SamplingParams(temperature=1.0, top_k=40), SamplingParams(temperature=1.0)]
    rng = random.Random(int(seed))
    return {"sampler": Sampler(get_library(DEVICE)), "logits": logits, "params": [kinds[i % len(kinds)] for i in range(R)],
            "seeds": [rng.randrange(1 << 31) for _ in range(R)], "index": [rng.randrange(512) for _ in range(R)]}


def run(state):
    if "sampler" in state:
        return state["sampler"].sample(state["logits"], state["params"], state["seeds"], state["index"])
    runner = state["runner"]
    out = torch.empty((state["rows"], state["vocab"]), dtype=torch.float32, device=DEVICE)
    row = 0
    for entries in state["steps"]:
        logits = runner.step(entries)
        if logits is not None:
            out[row:row + logits.shape[0]].copy_(logits)         # a decode step's logits are overwritten by the next one's
            row += logits.shape[0]
    for r in state["requests"]:
        runner.finish(r)
    return out


# ------------------------------------------------------------------------------------------- what it cannot do without
def _mixer_size(cfg, layer):
    """(multiply-adds per (query, key) pair, cached elements per key, window, elements of state, multiply-adds of the state per token)"""
    if "hidden_size" in cfg:
        return 2 * cfg["num_attention_heads"] * cfg["head_dim"], 2 * cfg["num_key_value_heads"] * cfg["head_dim"], None, 0, 0
    m, kind = layer["mixer"], layer["type"]
    if kind == "latent_attention":
        return m["heads"] * (2 * m["kv_rank"] + m["rot_dim"]), m["kv_rank"] + m["rot_dim"], None, 0, 0
    if kind == "attention":
        window = (m.get("mask") or {}).get("size")
        return 2 * m["heads"] * m["dim"], 2 * m["kv_heads"] * m["dim"], window, 0, 0
    if kind == "mamba2":
        s = m["heads"] * m["vdim"] * m["state"]
        return 0, 0, None, s, 3 * s
    if kind == "mamba1":
        s = m["inner"] * m["state"]
        return 0, 0, None, s, 3 * s
    if kind == "mlstm":
        s = m["heads"] * m["dim"] * m["vdim"]
        return 0, 0, None, s, 3 * s
    l, r = m["left"], m["right"]                                 # parallel: attention with mixed heads beside the delta rule
    s = r["heads"] * r["dim"] * r["vdim"]
    return 2 * l["heads"] * l["dim"] + l["heads"] ** 2, 2 * l["kv_heads"] * l["dim"], None, s, 4 * s


def work(case):
    """Every step streams the weights that its tokens need, the cached keys and values that its decoding requests see and the states
    of its requests once; every token takes the products of its weights, its attention and its state update."""
    if case["kind"] == "sample":
        return {"bytes": case["rows"] * (case["vocab"] * 4 + 4), "flops": 0}
    cfg = MODELS[case["model"]]()
    el = 4 if case["dtype"] == "float32" else 2
    specs = tensor_shapes(cfg)
    expert, fixed, head = 0, 0, 0
    for name, shape in specs.items():
        n = int(np.prod(shape)) if shape else 1
        part = name.split(".mlp.e")[1].split(".")[0] if ".mlp.e" in name else ""
        if part.isdigit():
            expert += n if part == "0" else 0
        elif name in ("model.embed_tokens.weight", "embed"):
            head = n if "lm_head.weight" not in specs and "head" not in specs else head
        elif name in ("lm_head.weight", "head"):
            head = n
        elif "table" in name or name == "side.embed":
            pass
        else:
            fixed += n
    layers = [None] * cfg["num_hidden_layers"] if "hidden_size" in cfg else cfg["layers"]
    times = (cfg.get("loop") or {}).get("times", 1)
    routers = [l["mlp"]["router"] for l in layers if l and l["mlp"]["kind"] == "moe"]
    experts, top = (routers[0]["experts"], routers[0]["top"]) if routers else (0, 0)
    total_bytes = total_flops = 0.0
    for step in plan(case):
        T = sum(k for _, _, k, _ in step)
        rows = sum(1 for e in step if e[3])
        used = experts * (1 - (1 - top / experts) ** T) if experts else 0
        total_bytes += times * (fixed + used * expert) * el + (head * el + rows * cfg_vocab(cfg) * 4 if rows else 0)
        total_flops += 2.0 * (times * T * (fixed + top * expert) + rows * head)
        for layer in layers:
            pair, kv, window, state, upd = _mixer_size(cfg, layer)
            for _, a, k, _ in step:
                seen = sum(min(p + 1, window or p + 1) for p in range(a, a + k)) if window else k * a + k * (k + 1) / 2
                total_flops += times * 2.0 * (pair * seen + upd * k)
                total_bytes += times * (kv * min(a + k, (window or a + k) + k - 1) * el + 2 * state * 4)
    return {"bytes": total_bytes, "flops": total_flops}


def cfg_vocab(cfg):
    return cfg["vocab_size"] if "hidden_size" in cfg else cfg["vocab"]


def tensor_shapes(cfg):
    return {n: s.shape for n, s in expected_tensors(config_from_dict(cfg).to_spec()).items()}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"                                           # every deciding sum is an integer or added in a fixed order
    if case["dtype"] == "float32":
        return {"rel": 3e-5}                                     # 9e-6 off 64 bits: sums of up to 18,944 products, four layers
    if case["model"].startswith("tugodra"):
        return {"rel": 0.03, "max": 0.9}                         # a near-tie of its router moves a token's logits by a tenth
    return {"rel": 0.03, "max": 0.3}                             # 0.004 to 0.019 off 64 bits: bfloat16 between the kernels of four layers


# --------------------------------------------------------------------------- the same in 64 bits, in plain array operations
def _unit(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def _silu(v):
    return v * torch.sigmoid(v)


def _gelu(v):
    return 0.5 * v * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (v + 0.044715 * v ** 3)))


def _angles(positions, dims, base, scaling=None):
    freq = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if scaling:
        low, high = scaling["original_max_position_embeddings"] / scaling["low_freq_factor"], scaling["original_max_position_embeddings"] / scaling["high_freq_factor"]
        for i, f in enumerate(freq):
            wave = 2.0 * math.pi / f
            s = (scaling["original_max_position_embeddings"] / wave - scaling["low_freq_factor"]) / (scaling["high_freq_factor"] - scaling["low_freq_factor"])
            freq[i] = f if wave < high else f / scaling["factor"] if wave > low else (1 - s) * f / scaling["factor"] + s * f
    ang = positions.to(F64)[:, None, None] * torch.tensor(freq, dtype=F64, device=DEVICE)
    return torch.cos(ang), torch.sin(ang)


def _turn(v, cs, dims, neighbours=False):
    """v [T, heads, D]: pairs (i, i + dims/2), or neighbours (2i, 2i + 1), of the leading `dims` elements turn."""
    c, s = cs
    out = v.clone()
    a, b = (v[..., 0:dims:2], v[..., 1:dims:2]) if neighbours else (v[..., :dims // 2], v[..., dims // 2:dims])
    x, y = a * c - b * s, b * c + a * s
    if neighbours:
        out[..., 0:dims:2], out[..., 1:dims:2] = x, y
    else:
        out[..., :dims // 2], out[..., dims // 2:dims] = x, y
    return out


def _attend(q, k, v, parts, scale, cap=None, sink=None, window=None, distance=None, talk=None, chunk=None):
    """Causal attention request by request: q [T, H, D], k [T, G, D], v [T, G, V]; query head h reads key head h // (H / G)."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty((q.shape[0], H, v.shape[2]), dtype=F64, device=DEVICE)
    for a, b in parts:
        block = max(1, min(b - a, (1 << 28) // (H * (b - a))))
        for i in range(a, b, block):
            e = min(b, i + block)
            s = torch.einsum("tgrd,jgd->grtj", q[i:e].reshape(e - i, G, H // G, -1), k[a:e]).reshape(H, e - i, e - a) * scale
            if cap is not None:
                s = cap * torch.tanh(s / cap)
            dist = torch.arange(i - a, e - a, device=DEVICE)[:, None] - torch.arange(e - a, device=DEVICE)[None, :]
            if distance is not None:
                s = s - distance[0][:, None, None] * torch.log1p(distance[1][:, None, None] * dist.clamp(min=0).to(F64))
            hidden = dist < 0
            if window is not None:
                hidden = hidden | (dist >= window)
            if chunk is not None:
                at = torch.arange(e - a, device=DEVICE) // chunk
                hidden = hidden | (at[i - a:][:, None] != at[None, :])
            s = s.masked_fill(hidden, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[:, None, None].expand(H, e - i, 1)], dim=2)
            p = torch.softmax(s, -1)[..., :e - a]
            if talk is not None:
                p = torch.einsum("hg,gtj->htj", talk, p)
            out[i:e] = torch.einsum("grtj,jgd->tgrd", p.reshape(G, H // G, e - i, e - a), v[a:e]).reshape(e - i, H, -1)
    return out


def _conv(u, taps, bias, parts):
    """Causal convolution per channel, the last tap on the current token, zeros before each request."""
    out = torch.empty_like(u)
    K = taps.shape[1]
    for a, b in parts:
        padded = torch.cat([torch.zeros((K - 1, u.shape[1]), dtype=F64, device=DEVICE), u[a:b]])
        out[a:b] = sum(padded[j:j + b - a] * taps[:, j] for j in range(K))
    return out if bias is None else out + bias


def _walk(parts, inputs, first, step):
    """Walk all requests side by side, token by token: `step(states, inputs of the tokens) -> (states, outputs)`."""
    n, longest = len(parts), max(b - a for a, b in parts)
    rows = torch.zeros((longest, n), dtype=torch.long, device=DEVICE)
    for r, (a, b) in enumerate(parts):
        rows[:b - a, r] = torch.arange(a, b, device=DEVICE)
    state, out = first(n), None
    for t in range(longest):
        state, y = step(state, [v[rows[t]] for v in inputs])
        if out is None:
            out = torch.empty((longest,) + y.shape, dtype=F64, device=DEVICE)
        out[t] = y
    return torch.cat([out[:b - a, r] for r, (a, b) in enumerate(parts)])


def _zeros(*shape):
    return torch.zeros(shape, dtype=F64, device=DEVICE)


def _dense_layer(x, W, i, cfg, pos, parts):
    H, G, D, p, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], f"model.layers.{i}.", cfg["rms_norm_eps"]
    d, ff, T = cfg["hidden_size"], cfg["intermediate_size"], x.shape[0]
    bias = cfg["architectures"][0].startswith("Qwen2")
    h = _unit(x, eps) * W(p + "input_layernorm.weight", (d,), "norm")
    q, k, v = [h @ W(f"{p}self_attn.{n}_proj.weight", (m * D, d)).T + (W(f"{p}self_attn.{n}_proj.bias", (m * D,), "bias") if bias else 0.0)
               for n, m in (("q", H), ("k", G), ("v", G))]
    cs = _angles(pos, D, cfg["rope_theta"], cfg.get("rope_scaling"))
    o = _attend(_turn(q.view(T, H, D), cs, D), _turn(k.view(T, G, D), cs, D), v.view(T, G, D), parts, D ** -0.5)
    x = x + o.reshape(T, -1) @ W(p + "self_attn.o_proj.weight", (d, H * D)).T
    h = _unit(x, eps) * W(p + "post_attention_layernorm.weight", (d,), "norm")
    y = _silu(h @ W(p + "mlp.gate_proj.weight", (ff, d)).T) * (h @ W(p + "mlp.up_proj.weight", (ff, d)).T)
    return x + y @ W(p + "mlp.down_proj.weight", (d, ff)).T


def _sink_attention(h, W, p, m, eps, pos, parts):
    T, d, H, G, D = h.shape[0], h.shape[1], m["heads"], m["kv_heads"], m["dim"]
    q, k = h @ W(p + "q", (H * D, d)).T, h @ W(p + "k", (G * D, d)).T
    cs = _angles(pos, m["rot"]["dims"], m["rot"]["base"])
    qn = _turn((_unit(q, eps) * W(p + "q.norm", (H * D,), "norm")).view(T, H, D), cs, m["rot"]["dims"])
    kn = _turn((_unit(k, eps) * W(p + "k.norm", (G * D,), "norm")).view(T, G, D), cs, m["rot"]["dims"])
    o = _attend(qn, kn, k.view(T, G, D), parts, m["scale"], cap=m["softcap"], sink=W(p + "sink", (H,), "bias"))
    o = o * torch.sigmoid(h @ W(p + "g", (H, d)).T)[:, :, None]
    return o.reshape(T, -1) @ W(p + "o", (d, H * D)).T


def _mamba2(h, W, p, m, eps, parts):
    T, d, H, P, N, G = h.shape[0], h.shape[1], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    z, u, dt = (h @ W(p + "in", (2 * inner + 2 * G * N + H, d)).T).split([inner, inner + 2 * G * N, H], dim=1)
    u = _silu(_conv(u, W(p + "conv", (inner + 2 * G * N, m["conv"]), "conv_taps"), W(p + "conv.b", (inner + 2 * G * N,), "bias"), parts))
    x, B, C = u[:, :inner].reshape(T, H, P), u[:, inner:inner + G * N].reshape(T, G, N), u[:, inner + G * N:].reshape(T, G, N)
    dt = torch.nn.functional.softplus(dt + W(p + "dt_bias", (H,), "bias"))
    keep = torch.exp(-torch.exp(W(p + "A_log", (H,), "bias")) * dt)

    def step(S, v):
        xt, Bt, Ct, dtt, kt = v
        Bt, Ct = Bt.repeat_interleave(H // G, dim=1), Ct.repeat_interleave(H // G, dim=1)
        S = kt[..., None, None] * S + (dtt[..., None] * xt)[..., None] * Bt[:, :, None, :]
        return S, (S @ Ct[..., None])[..., 0]
    y = _walk(parts, [x, B, C, dt, keep], lambda n: _zeros(n, H, P, N), step) + W(p + "D", (H,), "norm")[:, None] * x
    y = y.reshape(T, inner) * _silu(z)
    y = _unit(y.view(T, m["norm_groups"], -1), eps).reshape(T, inner) * W(p + "norm", (inner,), "norm")
    return y @ W(p + "o", (d, inner)).T


def _latent_attention(h, W, p, m, eps, pos, parts, neighbours, gate):
    T, d, H, D, R, V, rank = h.shape[0], h.shape[1], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    cs = _angles(pos, m["rot"]["dims"], m["rot"]["base"])
    q = (h @ W(p + "q", (H * (D + R), d)).T).view(T, H, D + R)
    down = h @ W(p + "dkv", (rank + R, d)).T
    c = _unit(down[:, :rank], eps) * W(p + "dkv.norm", (rank,), "norm")
    q = torch.cat([q[..., :D], _turn(q[..., D:], cs, m["rot"]["dims"], neighbours)], dim=2)
    shared = _turn(down[:, None, rank:], cs, m["rot"]["dims"], neighbours).expand(T, H, R)
    k = torch.cat([(c @ W(p + "uk", (H * D, rank)).T).view(T, H, D), shared], dim=2)
    v = (c @ W(p + "uv", (H * V, rank)).T).view(T, H, V)
    o = _attend(q, k, v, parts, m["scale"], sink=None if gate else W(p + "sink", (H,), "bias"))
    if gate:
        o = o * torch.sigmoid(h @ W(p + "g", (H, d)).T)[:, :, None]
    return o.reshape(T, -1) @ W(p + "o", (d, H * V)).T


def _experts(h, W, p, mlp, chosen, weights, f, names):
    """The sum over the chosen experts; `f` acts between an expert's first products and its last."""
    d, ff = h.shape[1], mlp["expert"]["ff"]
    out = torch.zeros_like(h)
    for e in range(mlp["router"]["experts"]):
        t, j = (chosen == e).nonzero(as_tuple=True)
        if len(t):
            y = f(*[h[t] @ W(f"{p}e{e}.{n}", (ff, d)).T for n in names]) @ W(f"{p}e{e}.down", (d, ff)).T
            out.index_add_(0, t, y * weights[t, j][:, None])
    return out


def _mixed_attention(h, W, p, m, eps, parts):
    T, d, H, G, D, V = h.shape[0], h.shape[1], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = [(h @ W(p + n, (a * b, d)).T + W(p + n + ".b", (a * b,), "bias")).view(T, a, b) for n, a, b in (("q", H, D), ("k", G, D), ("v", G, V))]
    r1, r2 = W(p + "r1", (H,), "coef"), W(p + "r2", (H,), "coef")
    o = _attend(q, k, _unit(v, eps), parts, m["scale"], distance=(r1, r2), talk=W(p + "talk", (H, H), "mixing"), chunk=m["mask"]["size"])
    return o.reshape(T, -1) @ W(p + "o", (d, H * V)).T + W(p + "o.b", (d,), "bias")


def _delta_rule(h, W, p, m, eps, parts):
    T, d, H, G, D, V = h.shape[0], h.shape[1], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = [_silu(_conv(h @ W(p + n, (a * b, d)).T, W(f"{p}{n}.conv", (a * b, m["conv"]), "conv_taps"), None, parts)).view(T, a, b)
               for n, a, b in (("q", G, D), ("k", G, D), ("v", H, V))]
    q, k = [(u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1) for u in (q, k)]
    beta = torch.sigmoid(h @ W(p + "b", (H, d)).T)
    keep = torch.exp(-torch.exp(W(p + "A_log", (H,), "bias")) * torch.nn.functional.softplus(h @ W(p + "a", (H, d)).T + W(p + "dt_bias", (H,), "bias")))

    def step(S, u):
        qt, kt, vt, bt, gt = u
        S = gt[..., None, None] * S
        S = S + kt[..., None] * (bt[..., None] * (vt - (kt[..., None, :] @ S)[..., 0, :]))[..., None, :]
        return S, (qt[..., None, :] @ S)[..., 0, :]
    o = _walk(parts, [q * D ** -0.5, k, v, beta, keep], lambda n: _zeros(n, H, D, V), step)
    o = _unit(o, eps) * W(p + "norm", (V,), "norm") * _silu(h @ W(p + "g", (H * V, d)).T).view(T, H, V)
    return o.reshape(T, -1) @ W(p + "o", (d, H * V)).T


def _mamba1(h, W, p, m, parts):
    d, inner, N, r = h.shape[1], m["inner"], m["state"], m["dt_rank"]
    u, z = (h @ W(p + "in", (2 * inner, d)).T).split(inner, dim=1)
    u = _silu(_conv(u, W(p + "conv", (inner, m["conv"]), "conv_taps"), W(p + "conv.b", (inner,), "bias"), parts))
    low, B, C = (u @ W(p + "x", (r + 2 * N, inner)).T).split([r, N, N], dim=1)
    dt = torch.nn.functional.softplus(low @ W(p + "dt", (inner, r)).T + W(p + "dt.b", (inner,), "bias"))
    A = -torch.exp(W(p + "A_log", (inner, N), "bias"))

    def step(S, v):
        ut, dtt, Bt, Ct = v
        S = torch.exp(dtt[..., None] * A) * S + (dtt * ut)[..., None] * Bt[:, None, :]
        return S, (S @ Ct[..., None])[..., 0]
    y = _walk(parts, [u, dt, B, C], lambda n: _zeros(n, inner, N), step) + W(p + "D", (inner,), "norm") * u
    return (y * _silu(z)) @ W(p + "o", (d, inner)).T


def _mlstm(h, W, p, m, eps, parts):
    T, d, H, D, V, cap = h.shape[0], h.shape[1], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = [(h @ W(p + n, (H * b, d)).T).view(T, H, b) for n, b in (("q", D), ("k", D), ("v", V))]
    gates = [cap * torch.tanh((h @ W(p + n, (H, d)).T + W(p + n + ".b", (H,), "bias")) / cap) for n in ("i", "f")]

    def step(state, u):
        S, n, top = state
        qt, kt, vt, take, keep = u
        new = torch.maximum(keep + top, take)
        keep, take = torch.exp(keep + top - new), torch.exp(take - new)
        S = keep[..., None, None] * S + take[..., None, None] * kt[..., None] * vt[..., None, :]
        n = keep[..., None] * n + take[..., None] * kt
        y = (qt[..., None, :] @ S)[..., 0, :] / (torch.maximum((n * qt).sum(-1).abs(), torch.exp(-new)) + 1e-6)[..., None]
        return (S, n, new), y
    y = _walk(parts, [q * D ** -0.5, k, v, gates[0], torch.nn.functional.logsigmoid(gates[1])], lambda n: (_zeros(n, H, D, V), _zeros(n, H, D), _zeros(n, H)), step)
    y = _unit(y, eps).reshape(T, H * V) * W(p + "norm", (H * V,), "norm") * torch.sigmoid(h @ W(p + "g", (H * V, d)).T)
    return y @ W(p + "o", (d, H * V)).T


def _exact_dense(cfg, W, ids, pos, parts):
    x = W("model.embed_tokens.weight", (cfg["vocab_size"], cfg["hidden_size"]))[ids]
    for i in range(cfg["num_hidden_layers"]):
        x = _dense_layer(x, W, i, cfg, pos, parts)
    x = _unit(x, cfg["rms_norm_eps"]) * W("model.norm.weight", (cfg["hidden_size"],), "norm")
    return x, W("model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight", (cfg["vocab_size"], cfg["hidden_size"]))


def _exact_tufirax(cfg, W, ids, pos, parts):
    d, eps = cfg["width"], cfg["norm"]["eps"]
    x = W("embed", (cfg["vocab"], d))[ids]
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        y = _sink_attention(x, W, p + "mix.", m, eps, pos, parts) if layer["type"] == "attention" else _mamba2(x, W, p + "mix.", m, eps, parts)
        x = x + _unit(y, eps) * W(p + "norm1", (d,), "norm")
        y = (_gelu(x @ W(p + "mlp.gate", (ff, d)).T) * (x @ W(p + "mlp.up", (ff, d)).T)) @ W(p + "mlp.down", (d, ff)).T
        x = x + _unit(y, eps) * W(p + "norm2", (d,), "norm")
    return _unit(x, eps) * W("final.norm", (d,), "norm"), W("head", (cfg["vocab"], d))


def _exact_vipelix(cfg, W, ids, pos, parts):
    d, eps, loop = cfg["width"], cfg["norm"]["eps"], cfg["loop"]
    embedded = W("embed", (cfg["vocab"], d))[ids]
    x = embedded
    for n in range(loop["times"]):
        x = x + (embedded if n else 0.0) + W("loop.step", (loop["times"], d), "bias")[n]
        for i, layer in enumerate(cfg["layers"]):
            p, mlp = f"l{i}.", layer["mlp"]
            y = _latent_attention(_unit(x, eps) * W(p + "norm1", (d,), "norm"), W, p + "mix.", layer["mixer"], eps, pos, parts, True, True)
            x = x + _unit(y, eps) * W(p + "norm1b", (d,), "norm")
            h = _unit(x, eps) * W(p + "norm2", (d,), "norm")
            p += "mlp."
            if mlp["kind"] == "dense":
                z, a = h @ W(p + "up", (mlp["ff"], d)).T, W(p + "act", (4,), "coef")
                z = a[0] * _unit(z, eps) + a[1] * _unit(z * z, eps) + a[2] * _unit(z ** 3, eps) + a[3]
                y = z @ W(p + "down", (d, mlp["ff"])).T
            else:
                top, s = mlp["router"]["top"], mlp["shared"]["ff"]
                chosen = W(p + "table", (cfg["vocab"], top), f"choice:{mlp['router']['experts']}")[ids].long()
                glu = lambda g, u: _silu(g) * u
                y = _experts(h, W, p, mlp, chosen, torch.full(chosen.shape, 1.0 / top, dtype=F64, device=DEVICE), glu, ("gate", "up"))
                y = y + glu(h @ W(p + "shared.gate", (s, d)).T, h @ W(p + "shared.up", (s, d)).T) @ W(p + "shared.down", (d, s)).T
            x = x + _unit(y, eps) * W(f"l{i}.norm2b", (d,), "norm")
    return _unit(x, eps) * W("final.norm", (d,), "norm"), W("embed", (cfg["vocab"], d))


def _exact_tibepel(cfg, W, ids, pos, parts):
    d, eps, side = cfg["width"], cfg["norm"]["eps"], cfg["token_side"]["dim"]
    norm = lambda v, name: _unit(v, eps) * (1.0 + W(name, (d,), "norm"))
    ang = pos.to(F64)[:, None] * torch.tensor([10000.0 ** (-2.0 * i / d) for i in range(d // 2)], dtype=F64, device=DEVICE)
    x = W("embed", (cfg["vocab"], d))[ids] * cfg["embedding"]["scale"] + torch.stack([torch.sin(ang), torch.cos(ang)], dim=2).reshape(-1, d)
    table = W("side.embed", (cfg["vocab"], len(cfg["layers"]) * side))
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        h = norm(x, p + "norm1")
        if layer["type"] == "mamba1":
            x = x + _mamba1(h, W, p + "mix.", m, parts)
        else:
            x = x + m["left_scale"] * _mixed_attention(h, W, p + "mix.left.", m["left"], eps, parts) + \
                m["right_scale"] * _delta_rule(h, W, p + "mix.right.", m["right"], eps, parts)
        h, q, ff, lim = norm(x, p + "norm2"), p + "mlp.", mlp["ff"], mlp["limit"]
        g = (h @ W(q + "gate", (ff, d)).T + W(q + "gate.b", (ff,), "bias")).clamp(max=lim)
        u = (h @ W(q + "up", (ff, d)).T + W(q + "up.b", (ff,), "bias")).clamp(-lim, lim)
        x = x + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W(q + "down", (d, ff)).T + W(q + "down.b", (d,), "bias")
        y = (_gelu(x @ W(p + "side.gate", (side, d)).T) * table[ids][:, i * side:(i + 1) * side]) @ W(p + "side.proj", (d, side)).T
        x = x + _unit(y, eps) * W(p + "side.norm", (d,), "norm")
    return norm(x, "final.norm"), W("head", (cfg["vocab"], d))


def _exact_tugodra(cfg, W, ids, pos, parts):
    d, eps = cfg["width"], cfg["norm"]["eps"]
    norm = lambda v, name: torch.tanh(W(name + ".alpha", (), "unit_scale") * v) * W(name, (d,), "norm") + W(name + ".b", (d,), "bias")
    x = W("embed", (cfg["vocab"], d))[ids] * cfg["embedding"]["scale"]
    T, kept = x.shape[0], {}
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp, q = f"l{i}.", layer["mixer"], layer["mlp"], f"l{i}.mix."
        h = norm(x, p + "norm1")
        if layer["type"] == "mlstm":
            y = _mlstm(h, W, q, m, eps, parts)
        elif layer["type"] == "latent_attention":
            y = _latent_attention(h, W, q, m, eps, pos, parts, False, False)
        else:
            H, G, D = m["heads"], m["kv_heads"], m["dim"]
            cs = _angles(pos, m["rot"]["dims"], m["rot"]["base"])
            if "kv_from" not in m:
                k = _turn((h @ W(q + "k", (G * D, d)).T).view(T, G, D), cs, m["rot"]["dims"], True)
                kept[i] = _unit(k, eps), (h @ W(q + "v", (G * D, d)).T).view(T, G, D)
            k, v = kept[m.get("kv_from", i)]
            u = _unit(_turn((h @ W(q + "q", (H * D, d)).T).view(T, H, D), cs, m["rot"]["dims"], True), eps)
            o = _attend(u, k, v, parts, m["scale"], window=m["mask"]["size"]) * torch.sigmoid(h @ W(q + "g", (H, d)).T)[:, :, None]
            y = o.reshape(T, -1) @ W(q + "o", (d, H * D)).T
        x = x + norm(y, p + "norm1b")
        h, q, r, s = norm(x, p + "norm2"), p + "mlp.", mlp["router"], mlp["shared"]["ff"]
        E, groups = r["experts"], r["groups"]
        score = torch.sigmoid(h @ W(q + "router", (E, d)).T)
        by_group = (score + W(q + "correction", (E,), "bias")).view(T, groups["count"], -1)
        best = by_group.topk(min(2, by_group.shape[2]), dim=2).values.sum(2).topk(groups["keep"], dim=1).indices
        allowed = torch.zeros((T, groups["count"]), dtype=torch.bool, device=DEVICE).scatter_(1, best, True)
        chosen = by_group.masked_fill(~allowed[:, :, None], float("-inf")).reshape(T, E).topk(r["top"], dim=1).indices
        weights = score.gather(1, chosen)
        squared = lambda u: torch.relu(u) ** 2
        y = _experts(h, W, q, mlp, chosen, weights / weights.sum(1, keepdim=True), squared, ("up",))
        gate = torch.sigmoid(h @ W(q + "shared.sg", (1, d)).T)
        y = y + gate * (squared(h @ W(q + "shared.up", (s, d)).T) @ W(q + "shared.down", (d, s)).T)
        x = x + norm(y, p + "norm2b")
    return norm(x, "final.norm"), W("head", (cfg["vocab"], d))


def exact(case, seed):
    if case["kind"] == "sample":
        return None                                              # drawn tokens: no value in 64 bits
    cfg = MODELS[case["model"]]()
    vocab = cfg_vocab(cfg)
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16

    def W(name, shape, init="matrix"):
        t = tensor(seed, name, shape, init, dtype)
        return t.to(F64) if t.is_floating_point() else t
    seqs = token_ids(case, seed, vocab)
    starts = np.cumsum([0] + [len(s) for s in seqs]).tolist()
    parts = list(zip(starts[:-1], starts[1:]))
    ids = torch.tensor([t for s in seqs for t in s], device=DEVICE)
    pos = torch.cat([torch.arange(len(s), device=DEVICE) for s in seqs])
    forward = {"llama": _exact_dense, "qwen": _exact_dense, "tufirax": _exact_tufirax, "vipelix": _exact_vipelix,
               "tibepel": _exact_tibepel, "tugodra": _exact_tugodra}[case["model"].split("-")[0]]
    x, head = forward(cfg, W, ids, pos, parts)
    wanted = [starts[r] + a + k - 1 for step in plan(case) for r, a, k, want in step if want]
    logits = x[torch.tensor(wanted, device=DEVICE)] @ head.T
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits
