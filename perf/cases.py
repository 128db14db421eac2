"""What a user of the library has it do, as cases that can be timed and compared.

A pass serves one batch of requests: the prompts go in as one step, every later step carries one token of each sequence (the
token sampled before it), and a last step returns the logits behind everything that was generated.  A case without new
tokens is one step that returns the logits behind its prompts.  The sizes are those of the benchmark: the layer sizes of the
1B, 8B and 13B Llama configurations and the three size sets of the six other designs, in bfloat16 and in true float32.

Weights are drawn by tensor name, scaled so that activations stay of size one through all layers.  The embedding is a large
part of the residual and the output matrix holds it shifted by a few rows (or is the embedding itself), so that, as in a
trained model, the next token is a clear choice; routers answer to a part of the embedding that tokens of one group share,
so that experts are chosen clearly and unevenly.  Otherwise rounding would decide tokens and experts, and two correct
implementations could not be compared.

``exact`` restates the designs in plain torch in 64 bits: whole sequences, no cache, no batch.
"""
import math
import zlib

import numpy as np
import torch

import bitnet_c_b200 as bn
from bitnet_c_b200.config import architecture_of
from bitnet_c_b200.engine import Model, ModelEngine
from bitnet_c_b200.engine.model import parameter_table

DEVICE = "cuda:0"
SHIFT = 7  # with an output matrix of its own, token t + SHIFT follows token t
GROUPS = 64  # groups of tokens that routers tell apart

LLAMA = {  # width, heads, key/value heads, head size, feed-forward, layers, vocabulary, tied, rotary base, longest context
    "1b": (2048, 32, 8, 64, 8192, 16, 128256, True, 500000.0, 8192),
    "8b": (4096, 32, 8, 128, 14336, 32, 128256, False, 500000.0, 4096),
    "13b": (5120, 40, 40, 128, 13824, 40, 32000, False, 10000.0, 4096),
}
WIDTHS = {"w1024": 1024, "w2048": 2048, "w4096": 4096}
DESIGNS = ("fesorax", "lotilix", "mekevik", "netanex", "rudolix", "lakadra")


# ---- cases --------------------------------------------------------------------------------------------------------
def listed():
    def case(name, design, size, batch, longest, new, **more):
        return dict({"name": name, "design": design, "size": size, "dtype": "bfloat16", "batch": batch, "longest": longest,
                     "ragged": False, "new": new, "temperature": 0.0, "layers": 0}, **more)

    return [
        # a short question to a small model and the first words of the answer: launches and latency
        case("llama-1b short reply", "llama", "1b", 1, 12, 8),
        # one user with a long prompt: the 2,048-token prefill, then decode at batch 1
        case("llama-8b long prompt", "llama", "8b", 1, 2048, 16),
        # a small batch of requests: decode at batch 8, the benchmark's main number
        case("llama-8b batch of 8", "llama", "8b", 8, 512, 32),
        # serving many users: 64 prompts of any length as one ragged step, decode at batch 64, nucleus sampling
        case("llama-1b batch of 64", "llama", "1b", 64, 2048, 32, ragged=True, temperature=0.7),
        # the largest weights, no grouped heads, unequal lengths
        case("llama-13b unequal", "llama", "13b", 8, 2048, 32, ragged=True),
        # true single precision, a quarter of the layers as in the benchmark
        case("llama-8b float32", "llama", "8b", 8, 65, 16, dtype="float32", layers=8),
        # the other designs: each with prompts and generation, at sizes and batches spread over their size sets
        case("fesorax requests", "fesorax", "w2048", 4, 2048, 32, ragged=True),
        case("lotilix long prompt", "lotilix", "w2048", 1, 2011, 32),
        case("mekevik batch", "mekevik", "w4096", 8, 300, 32),
        case("netanex two long", "netanex", "w4096", 2, 4000, 16, ragged=True),
        case("rudolix small batch", "rudolix", "w1024", 16, 512, 48, ragged=True),
        case("lakadra requests", "lakadra", "w2048", 8, 1000, 32, ragged=True),
    ]


def cost(case):
    """Seconds a pass takes at rates a good implementation reaches: what keeps drawn cases below the largest listed one."""
    w = work(case)
    return w["bytes"] / 4e12 + w["flops"] / (6e14 if case["dtype"] == "bfloat16" else 5e13) + 2e-4 * (case["new"] + 2)


def draw(rng):
    most = max(cost(c) for c in listed())
    while True:
        design = rng.choice(("llama",) * 6 + DESIGNS)
        size = rng.choice(sorted(LLAMA) if design == "llama" else sorted(WIDTHS))
        dtype = "float32" if rng.random() < 0.12 and size in ("1b", "w1024", "w2048") else "bfloat16"
        case = {"design": design, "size": size, "dtype": dtype, "batch": round(math.exp(rng.uniform(0.0, math.log(64.5)))),
                "longest": round(math.exp(rng.uniform(math.log(3), math.log(4000)))), "ragged": rng.random() < 0.5,
                "new": rng.choice((0, rng.randint(1, 48), rng.randint(8, 48))), "layers": 0,
                "temperature": 0.7 if rng.random() < 0.2 else 0.0}
        if not case["new"]:
            case["temperature"] = 0.0
        if case["batch"] * case["longest"] <= (70000 if dtype == "bfloat16" else 8000) and cost(case) <= most:
            return case


# ---- configurations -------------------------------------------------------------------------------------------------
def config(case):
    size, design = case["size"], case["design"]
    if design == "llama":
        w, heads, kv, dim, ff, layers, vocab, tied, base, longest = LLAMA[size]
        return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_size": w, "intermediate_size": ff,
                "num_hidden_layers": case["layers"] or layers, "num_attention_heads": heads, "num_key_value_heads": kv,
                "head_dim": dim, "vocab_size": vocab, "max_position_embeddings": longest, "rope_theta": base,
                "rms_norm_eps": 1e-5, "tie_word_embeddings": tied, "hidden_act": "silu"}
    w = WIDTHS[size]
    big, heads, kv, dim, d, window = w == 4096, w // 128, w // 512, 128, 128, 1024
    ff = 14336 if big else 4 * w
    cfg = {"architecture": design.capitalize(), "vocab": 32000, "width": w, "norm": {"eps": 1e-6}, "max_positions": 8192}

    def layers(*pairs):
        return [dict({"type": t, "mixer": m, "mlp": mlp}, **more) for t, m, mlp, more in pairs]

    if design == "fesorax":
        att = {"heads": heads, "kv_heads": kv, "dim": d, "vdim": d, "scale": d ** -0.5 * 4, "bias_max": 4 * window,
               "mask": {"size": window, "keep_first": 64}}
        mem = {"heads": w // 256, "dim": 128, "vdim": 256, "gate_cap": 15.0}
        mlp = {"kind": "moe", "router": {"experts": 8 if w == 1024 else 16, "top": 2}, "expert": {"ff": w // 2, "limit": 7.0},
               "shared": {"ff": w, "limit": 7.0}}
        return dict(cfg, postln_alpha=2.0, embedding={"scale": 1.0}, layers=layers(
            ("attention", att, mlp, {}), ("mlstm", mem, mlp, {}), ("attention", dict(att, kv_from=0), mlp, {}), ("attention", att, mlp, {})))
    rank = 512 if big else 192
    latent = {"heads": heads, "dim": d, "rot_dim": 64, "vdim": d, "q_rank": 3 * w // 8, "kv_rank": rank, "scale": (d + 64) ** -0.5,
              "rot": {"base": 1e6, "dims": 64}}
    delta = {"heads": heads, "kv_heads": heads, "dim": d, "vdim": d, "conv": 4}
    half = {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": ff // 2}}
    if design == "lotilix":
        low = 128 if big else 64
        att = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "mask": {"size": window},
               "rot": {"base": 5e5, "dims": dim, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        seen, mlp = dict(latent, mask={"size": window}), {"kind": "dense", "ff": ff}
        return dict(cfg, token_side={"dim": 128 if w == 1024 else 256}, layers=layers(
            ("latent_attention", seen, mlp, {}), ("channel_delta", dict(delta, decay_rank=low, gate_rank=low), mlp, {}),
            ("attention", att, mlp, {}), ("latent_attention", seen, mlp, {})))
    if design == "mekevik":
        att = {"heads": heads, "kv_heads": kv, "dim": d, "vdim": d, "scale": d ** -0.5 * 4, "bias_max": 4 * window,
               "mask": {"size": window}, "v_mix": True}
        dense = {"kind": "dense", "ff": ff, "limit": 7.0}
        moe = dict(half, router={"experts": 8, "top": 2, "scale": 1.0})
        return dict(cfg, embedding={"scale": 1.0}, logit_scale=1.0, layers=layers(*[("attention", att, m, {}) for m in (dense, moe, dense, moe)]))
    if design == "netanex":
        whole = {"heads": heads, "kv_heads": kv, "dim": d, "vdim": d, "scale": d ** -0.5 * 4}
        two = {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": d, "scale": 64 ** -0.5 * 4, "diff": 0.6, "q_temp": {"coef": 0.5, "every": 128}}
        lat = {k: v for k, v in latent.items() if k != "q_rank"}
        lat.update(mask={"size": window}, rot={"base": 1e6, "dims": 64, "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}})
        return dict(cfg, layers=layers(("attention_2", whole, half, {}), ("attention", two, half, {}), ("latent_attention", lat, half, {}),
                                       ("attention_2", whole, half, {"weights_of": 0})))
    if design == "rudolix":
        dense, moe = {"kind": "dense", "ff": ff}, dict(half, expert={"ff": ff // 2, "limit": 7.0})
        mamba = {"heads": w // 32, "groups": 1, "state": 128, "vdim": 64, "conv": 4, "norm_groups": 1}
        att = {"heads": heads, "kv_heads": kv, "dim": d, "vdim": d, "scale": d ** -0.5, "rot": {"base": 5e5, "dims": d}}
        return dict(cfg, streams=2, residual_mult=0.5, canon={"taps": 4}, embedding={"scale": 1.0}, layers=layers(
            ("mamba2", mamba, dense, {}), ("delta", delta, moe, {}), ("attention", att, dense, {}), ("mamba2", mamba, moe, {})))
    lightning = {"heads": heads, "dim": d, "vdim": d, "decay": [1.0 - 2.0 ** (-3.0 - 5.0 * h / heads) for h in range(heads)]}
    pair = {"left_scale": 0.5, "right_scale": 0.5,
            "left": {"heads": heads, "kv_heads": kv, "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": window},
                     "rot": {"base": 5e5, "dims": d, "scaling": {"factor": 8.0}}},
            "right": {"width": w, "blocks": min(heads, 16), "conv": 4}}
    mlp = {"kind": "moe", "router": {"experts": 14, "top": 2, "identity": 2, "groups": {"count": 4, "keep": 2}},
           "expert": {"ff": ff // 4}, "shared": {"ff": ff // 2}}
    return dict(cfg, logit_scale=1.0, logit_softcap=30.0, layers=layers(
        ("lightning", lightning, mlp, {}), ("latent_attention", latent, mlp, {}), ("parallel", pair, mlp, {}),
        ("latent_attention", dict(latent, kv_from=1), mlp, {})))


def vocabulary(cfg):
    return cfg.get("vocab") or cfg["vocab_size"]


def tied(cfg):
    return bool(cfg.get("tie_word_embeddings")) or cfg.get("architecture") in ("Netanex", "Rudolix")


def lengths(case, seed):
    """The prompts' lengths: all alike, or from one token to the longest, one of them the longest."""
    n, longest = case["batch"], case["longest"]
    if not case["ragged"]:
        return [longest] * n
    rng = np.random.default_rng(1000 + n)  # the same for every seed: another seed changes the tokens, not the work
    return [longest] + [int(v) for v in rng.integers(1, longest + 1, n - 1)]


def prompts(case, cfg, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, vocabulary(cfg), n).tolist() for n in lengths(case, seed)]


# ---- weights ----------------------------------------------------------------------------------------------------------
def shapes(cfg):
    """Every tensor of the model's file: name -> (shape, how it is filled, bound of its integers)."""
    arch = architecture_of(cfg)
    spec = arch.to_spec(arch.read_config(cfg))
    table = {path: (arch.tensor_name(path), p) for path, p in parameter_table(spec).items() if p.init != "unused"}
    return arch, spec, table


def drawn(name, seed):
    return torch.Generator(device=DEVICE).manual_seed((zlib.crc32(name.encode()) * 1000003 + seed * 7919) % (1 << 62))


def weights(cfg, seed, dtype):
    """The model's tensors by their names in the file."""
    _arch, _spec, table = shapes(cfg)
    n_layers = len(cfg["layers"]) if "layers" in cfg else cfg["num_hidden_layers"]
    out, width = {}, cfg.get("width") or cfg["hidden_size"]
    group = torch.randn(GROUPS, width, device=DEVICE, generator=drawn("groups", seed))

    def normal(name, shape, std, mean=0.0):
        t = torch.empty(shape, dtype=dtype, device=DEVICE)
        return t.normal_(mean, std, generator=drawn(name, seed))

    def uniform(name, shape, low, high):
        return torch.rand(shape, device=DEVICE, generator=drawn(name, seed)) * (high - low) + low

    for _path, (name, p) in table.items():
        if name in out:
            continue
        shape, last = tuple(p.shape), name.rsplit(".", 1)[-1]
        if name in ("embed", "model.embed_tokens.weight"):
            t = normal(name, shape, 0.8).float() + 0.6 * group[torch.arange(shape[0], device=DEVICE) % GROUPS]
            out[name] = (t * (0.2 if tied(cfg) else 1.0)).to(dtype)
        elif name in ("head", "lm_head.weight"):
            out[name] = (out["embed" if "embed" in out else "model.embed_tokens.weight"].float().roll(SHIFT, 0) * (1.5 / math.sqrt(width))).to(dtype)
        elif p.init == "distinct":
            out[name] = torch.rand(shape[0], p.high, device=DEVICE, generator=drawn(name, seed)).argsort(1)[:, :shape[1]].to(torch.int32).contiguous()
        elif last == "router":  # two experts stand out for the tokens of a group, others for another group's
            level = 0.3 * torch.randn(shape[0], GROUPS, device=DEVICE, generator=drawn(name, seed))
            best = torch.rand(shape[0], GROUPS, device=DEVICE, generator=drawn(name + "/", seed)).argsort(0)[:2]
            level.scatter_(0, best, torch.tensor([[4.0], [3.5]], device=DEVICE).expand(2, GROUPS))
            out[name] = (level @ group / (0.6 * width)).to(dtype)
        elif last in ("norm1b", "norm2b"):  # norms behind a sublayer, stored as the distance from one: they keep it small
            out[name] = normal(name, shape, 0.1, -0.7)
        elif p.init in ("ones", "around_zero"):
            out[name] = normal(name, shape, 0.1, 1.0 if p.init == "ones" else 0.0)
        elif p.init == "identity" or last == "talk":
            out[name] = (torch.eye(shape[0], device=DEVICE) + normal(name, shape, 0.1).float()).to(dtype)
        elif last == "A_log":
            out[name] = uniform(name, shape, 1.0, 16.0).log().to(dtype)
        elif last == "dt_bias":  # steps between a thousandth and a tenth
            out[name] = uniform(name, shape, math.log(1e-3), math.log(1e-1)).exp().expm1().log().to(dtype)
        elif last == "lam":  # decays that remember some ten to some thousand tokens
            out[name] = uniform(name, shape, math.log(5e-4), math.log(2e-2)).exp().expm1().log().to(dtype)
        elif last == "act":
            out[name] = (torch.tensor([0.4, 0.3, 0.2, 0.1], device=DEVICE)).to(dtype)
        elif last == "vmix":
            out[name] = torch.full(shape, 0.5, dtype=dtype, device=DEVICE)
        elif last == "pb":  # weights that are not normalised: about the logarithm of one over the window
            out[name] = normal(name, shape, 0.5, -6.5)
        elif name.endswith("f.b"):
            out[name] = normal(name, shape, 1.0, 3.0)
        elif last == "D":
            out[name] = normal(name, shape, 0.1, 1.0)
        elif last == "correction":
            out[name] = normal(name, shape, 0.02)
        elif last == "rel":
            out[name] = normal(name, shape, 0.5)
        elif last in ("canon1", "canon2", "lq1", "lk1", "lq2", "lk2", "b") and len(shape) < 3 and shape[-1] != width:
            out[name] = normal(name, shape, 0.1)
        elif len(shape) == 1 or (len(shape) == 2 and name.split(".")[-2] in ("ra", "ri")):
            out[name] = normal(name, shape, 1.0 if last == "sink" else 0.1)
        elif last == "conv":
            out[name] = normal(name, shape, 0.5)
        elif name == "side.embed":
            out[name] = normal(name, shape, 1.0)
        else:  # a matrix [out, in]; what is added to the residual is kept smaller the deeper the model is
            adds = last in ("o", "down", "proj") or ".o_proj." in name or ".down_proj." in name
            out[name] = normal(name, shape, (1.0 / math.sqrt(2 * n_layers) if adds else 1.0) / math.sqrt(shape[-1]))
    return out


# ---- one pass -----------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    """A loaded model with a cache and an engine for the batch, and the prompts as lists of token ids."""
    cfg = config(case)
    arch, spec, table = shapes(cfg)
    dtype = {"bfloat16": torch.bfloat16, "float32": torch.float32}[case["dtype"]]
    by_name = weights(cfg, seed, dtype)
    model = Model(spec, dtype=case["dtype"], device=DEVICE, arch=arch, config=arch.read_config(cfg))
    model.bind({path: by_name[name] for path, (name, _p) in table.items()})
    asked = prompts(case, cfg, seed)
    room = sum(-(-(len(p) + case["new"] + 1) // 64) * 64 for p in asked)
    cache = model.new_cache(max_tokens=room, max_seqs=len(asked))
    engine = ModelEngine(model, cache, bn.SamplingParams(temperature=case["temperature"], top_p=0.9, seed=seed))
    return {"model": model, "cache": cache, "engine": engine, "prompts": asked, "new": case["new"]}


def run(state):
    model, cache, engine, asked = state["model"], state["cache"], state["engine"], state["prompts"]
    rows = list(range(len(asked)))
    feed, tokens = asked, []
    if state["new"]:
        engine.start_batch(0, asked)
    slots = [engine.open() for _ in asked]
    for _ in range(state["new"]):
        sampled = engine.step_and_sample([bn.SeqStep(s, f, [len(f) - 1]) for s, f in zip(slots, feed)], rows)
        tokens.append(sampled)
        feed = [[t] for t in sampled]
    logits = model.step(cache, [bn.SeqStep(s, f, [len(f) - 1]) for s, f in zip(slots, feed)])
    for s in slots:
        engine.close(s)
    return {"tokens": np.asarray(tokens, dtype=np.int32), "logits": logits} if tokens else {"logits": logits}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def work(case):
    """The prompts' products and attention; for every single-token step one read of the weights it uses and of the cached
    rows and states it sees (a step's input is the step before's output, and the weights do not fit on the chip)."""
    cfg = config(case)
    _arch, _spec, table = shapes(cfg)
    item = 2 if case["dtype"] == "bfloat16" else 4
    lens, new = lengths(case, 0), case["new"]
    T, B, width, vocab = sum(lens), len(lens), cfg.get("width") or cfg["hidden_size"], vocabulary(cfg)
    dense = expert = n_experts = top = 0
    seen = set()
    for _path, (name, p) in table.items():
        n = math.prod(p.shape)
        if name in seen or name in ("embed", "head", "side.embed", "lm_head.weight", "model.embed_tokens.weight") or p.init == "distinct":
            continue
        seen.add(name)
        if ".mlp.e" in name:
            expert += n
        else:
            dense += n
    mixers = []  # per layer: query heads, key/value heads, key size, value size, window
    for layer in cfg.get("layers", [{"mixer": None}] * cfg.get("num_hidden_layers", 0)):
        m = layer["mixer"]
        if m is None:
            mixers.append((cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["head_dim"], 0))
            continue
        m = m.get("left", m)
        ro = (layer.get("mlp") or {}).get("router")
        if ro:
            n_experts, top = ro["experts"], ro["top"]
        if "kv_rank" in m:  # cached as one row for all heads
            mixers.append((m["heads"], 0, m["kv_rank"] + m["rot_dim"], m["vdim"], (m.get("mask") or {}).get("size", 0)))
        elif "scale" in m:
            mixers.append((m["heads"], m["kv_heads"], m["dim"] * (2 if "diff" in m else 1), m["vdim"], (m.get("mask") or {}).get("size", 0)))
        else:  # a state of keys x values per head: each token reads and changes it
            mixers.append((m["heads"], -1, m.get("dim") or m["state"], m["vdim"], 0))

    def touched(tokens):
        return expert * (1.0 - (1.0 - top / n_experts) ** tokens) if n_experts else 0.0

    step_flops = 2 * B * (dense + (expert * top / n_experts if n_experts else 0)) + 2.0 * B * vocab * width
    head = vocab * width * item + 4 * B * vocab
    flops = 2.0 * T * (dense + (expert * top / n_experts if n_experts else 0)) + 2.0 * B * vocab * width + new * step_flops
    moved = (dense + touched(T)) * item + head + T * width * item + new * ((dense + touched(B)) * item + head + B * width * item)
    for heads, kv, dk, dv, window in mixers:
        row = (dk if kv == 0 else kv * (dk + dv)) * item
        for n in lens:
            if kv < 0:
                flops += 6.0 * heads * dk * dv * (n + new)
                moved += 4 * heads * dk * dv * (1 + 2 * new)
                continue
            w = window or n + new + 1
            pairs = sum(min(p + 1, w) for p in range(n)) if window else n * (n + 1) / 2
            behind = sum(min(n + i + 1, w) for i in range(new))
            flops += 2.0 * heads * (dk + (dk if kv == 0 else dv)) * (pairs + behind)
            moved += row * (n + new + behind)
    return {"bytes": float(moved), "flops": float(flops)}


# Four times the relative error against ``exact`` that was seen over some fifty cases (single precision: 1.4e-6 at most).
TOLERANCE = {"1b": 0.02, "8b": 0.004, "13b": 0.004, "fesorax": 0.02, "lotilix": 0.014, "mekevik": 0.02, "netanex": 0.014,
             "rudolix": 0.02, "lakadra": 0.008}


def tolerance(case):
    rel = 6e-6 if case["dtype"] == "float32" else TOLERANCE[case["size"] if case["design"] == "llama" else case["design"]]
    return {"rel": rel, "max": 8 * rel, "differ": 0.005}


# ---- the designs in 64 bits ---------------------------------------------------------------------------------------------------
def exact(case, seed):
    if cost(case) > 1.0:
        return None
    cfg = config(case)
    w = weights(cfg, seed, {"bfloat16": torch.bfloat16, "float32": torch.float32}[case["dtype"]])
    step = 0 if tied(cfg) else SHIFT
    tokens, logits = [], []
    for p in prompts(case, cfg, seed):
        line = list(p)
        for _ in range(case["new"]):
            line.append((line[-1] + step) % vocabulary(cfg))
        z = Plain(cfg, w).logits(line, len(p) - 1)
        tokens.append([int(t) for t in z[:-1].argmax(1)] if case["new"] else [])
        if case["new"] and tokens[-1] != line[len(p):]:
            return None  # the line that was assumed is not the one that would be generated
        logits.append(z[-1])
    out = {"logits": torch.stack(logits)}
    if case["new"]:
        out["tokens"] = np.asarray(tokens, dtype=np.int32).T.copy()
    return out


def unit(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def unit_vector(x):
    return x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def limited(g, u, limit):
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


silu, sigmoid, softplus = torch.nn.functional.silu, torch.sigmoid, lambda z: torch.logaddexp(z, torch.zeros_like(z))


def convolution(x, taps, bias=0.0):
    n = taps.shape[1]
    past = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(past[j:j + x.shape[0]] * taps[:, j] for j in range(n)) + bias


def turned(x, angles, halves, size=1.0):
    """The first numbers of every head turned: number i with i + n / 2 (``halves``) or 2i with 2i + 1."""
    half = angles.shape[1]
    at_u = torch.arange(half, device=x.device) * (1 if halves else 2)
    at_v = at_u + (half if halves else 1)
    c, s = angles.cos()[:, None] * size, angles.sin()[:, None] * size
    out = x.clone()
    out[..., at_u], out[..., at_v] = x[..., at_u] * c - x[..., at_v] * s, x[..., at_v] * c + x[..., at_u] * s
    return out


def attend(q, k, v, scale, window=0, keep=0, chunk=0, sink=None, bias=None):
    """Softmax attention, q [T, H, d], k [T, G, d], v [T, G, dv]; ``sink`` one score per head in the denominator, ``bias``
    [distance, head]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device=q.device)
    apart = i[:, None] - i[None]
    seen = apart >= 0
    if window:
        seen &= (apart < window) | (i[None] < keep)
    if chunk:
        seen &= (i[:, None] // chunk) == (i[None] // chunk)
    out = q.new_empty(T, H, v.shape[2])
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        if bias is not None:
            s += bias[apart.clamp(min=0), h]
        s = s.masked_fill(~seen, -math.inf)
        top = s.amax(1, keepdim=True)
        if sink is not None:
            top = top.clamp(min=float(sink[h]))
        e = torch.exp(s - top)
        out[:, h] = e @ v[:, h * G // H] / (e.sum(1, keepdim=True) + (torch.exp(float(sink[h]) - top) if sink is not None else 0.0))
    return out


def buckets(T, count, most, like, single):
    """The bias bucket of every distance: one each below half the table, then by their logarithm."""
    n, half = np.arange(T), count // 2
    kind = np.float32 if single else np.float64
    far = np.log(np.maximum(n, half).astype(kind) / kind(half)) / kind(math.log(most / half))
    b = np.minimum(count - 1, half + np.floor(far.astype(kind) * kind(count - half)).astype(np.int64))
    return torch.from_numpy(np.where(n < half, n, b)).to(like.device)


def delta_rule(q, k, v, g, beta):
    """q, k [T, H, d], v [T, H, dv], g [T, H, d] or [T, H, 1], beta [T, H]."""
    S, out = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * g[t, :, :, None]
        u = beta[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
        S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
        out[t] = (q[t, :, None] @ S)[:, 0]
    return out


def state_sums(q, k, v, g):
    """S_t = g_t S_(t-1) + k_t v_t^T, read by q_t; g [T, H]."""
    S, out = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(q.shape[0]):
        S = torch.baddbmm(S * g[t, :, None, None], k[t, :, :, None], v[t, :, None])
        out[t] = (q[t, :, None] @ S)[:, 0]
    return out


class Plain:
    """One sequence through a design, from its first token."""

    def __init__(self, cfg, w):
        self.cfg, self.raw = cfg, w

    def w(self, name):
        return self.raw[name].double()

    def lin(self, x, name):
        return x @ self.w(name).T

    def heads(self, x, name, n):
        return self.lin(x, name).reshape(x.shape[0], n, -1)

    def norm(self, x, name, one=0.0):
        return unit(x, self.eps) * (one + self.w(name))

    def logits(self, tokens, first):
        """Logits at positions ``first`` to the end."""
        t = torch.tensor(tokens, device=DEVICE)
        self.eps = self.cfg["norm"]["eps"] if "norm" in self.cfg else self.cfg["rms_norm_eps"]
        self.kept = {}
        return getattr(self, self.cfg.get("architecture", "Llama").lower())(t, first)

    # -- Llama
    def llama(self, t, first):
        c = self.cfg
        H, G, d = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        step = np.power(np.float32(c["rope_theta"]), np.float32(-2.0) / np.float32(d)).astype(np.float32)
        a = np.empty((len(t), d // 2), dtype=np.float32)  # the angles are a running product in single precision
        a[:, 0] = np.arange(len(t))
        for i in range(1, d // 2):
            a[:, i] = a[:, i - 1] * step
        a = torch.from_numpy(a).to(DEVICE).double()
        x = self.raw["model.embed_tokens.weight"][t].double()
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = self.norm(x, p + "input_layernorm.weight")
            q, k, v = (self.heads(h, f"{p}self_attn.{n}_proj.weight", m) for n, m in (("q", H), ("k", G), ("v", G)))
            o = attend(turned(q, a, True), turned(k, a, True), v, d ** -0.5)
            x = x + self.lin(o.flatten(1), p + "self_attn.o_proj.weight")
            h = self.norm(x, p + "post_attention_layernorm.weight")
            x = x + self.lin(silu(self.lin(h, p + "mlp.gate_proj.weight")) * self.lin(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
        return self.lin(self.norm(x[first:], "model.norm.weight"), "lm_head.weight" if "lm_head.weight" in self.raw else "model.embed_tokens.weight")

    # -- experts: ids and weights [T, top]; the result of each chosen expert times its weight
    def experts(self, h, ids, weight, unit_of, scaled_input=False):
        out = torch.zeros_like(h)
        for e in range(int(ids.max()) + 1):
            rows, place = (ids == e).nonzero(as_tuple=True)
            if len(rows):
                s = weight[rows, place][:, None]
                out[rows] += unit_of(h[rows] * s, e) if scaled_input else s * unit_of(h[rows], e)
        return out

    def gated(self, h, p, act):
        return self.lin(act(self.lin(h, p + "gate"), self.lin(h, p + "up")), p + "down")

    # -- Fesorax
    def fesorax(self, t, first):
        c, eps = self.cfg, self.eps
        x = self.raw["embed"][t].double() * c["embedding"]["scale"]
        for i, L in enumerate(c["layers"]):
            p, m, f = f"l{i}.mix.", L["mixer"], L["mlp"]
            H = m["heads"]
            if L["type"] == "attention":
                if m.get("kv_from") is None:
                    self.kept[i] = unit(self.heads(x, p + "k", m["kv_heads"]), eps), self.heads(x, p + "v", m["kv_heads"])
                k, v = self.kept[m.get("kv_from", i)]
                rel = self.w(p + "rel")
                bias = rel[buckets(len(t), rel.shape[0], m["bias_max"], rel, True)]
                o = attend(unit(self.heads(x, p + "q", H), eps), k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], bias=bias)
                y = (o * sigmoid(self.lin(x, p + "g"))[:, :, None]).flatten(1)
            else:
                cap = m["gate_cap"]
                q, k, v = (self.heads(x, p + n, H) for n in "qkv")
                gi = cap * torch.tanh((self.lin(x, p + "i") + self.w(p + "i.b")) / cap)
                gf = -softplus(-cap * torch.tanh((self.lin(x, p + "f") + self.w(p + "f.b")) / cap))
                y = unit(self.memory(q * m["dim"] ** -0.5, k, v, gi, gf), eps).flatten(1) * self.w(p + "norm") * sigmoid(self.lin(x, p + "g"))
            x = self.norm(c["postln_alpha"] * x + self.lin(y, p + "o"), f"l{i}.norm1")
            p = f"l{i}.mlp."
            s, ids = sigmoid(self.lin(x, p + "router")).topk(f["router"]["top"])
            y = self.experts(x, ids, s, lambda a, e: self.gated(a, f"{p}e{e}.", lambda g, u: limited(g, u, f["expert"]["limit"])), True)
            y = y + self.gated(x, p + "shared.", lambda g, u: limited(g, u, f["shared"]["limit"]))
            x = self.norm(c["postln_alpha"] * x + y, f"l{i}.norm2")
        return self.lin(self.norm(x[first:], "final.norm"), "head")

    def memory(self, q, k, v, gi, gf):
        """A matrix memory per head under stabilised exponential gates."""
        S, n = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), q.new_zeros(q.shape[1], q.shape[2])
        top, out = q.new_zeros(q.shape[1]), torch.empty_like(v)
        for t in range(q.shape[0]):
            new = torch.maximum(gf[t] + top, gi[t])
            a, b, top = torch.exp(gf[t] + top - new), torch.exp(gi[t] - new), new
            S = torch.baddbmm(S * a[:, None, None], (k[t] * b[:, None])[:, :, None], v[t, :, None])
            n = n * a[:, None] + k[t] * b[:, None]
            out[t] = (q[t, :, None] @ S)[:, 0] / (torch.maximum((n * q[t]).sum(1).abs(), torch.exp(-top)) + 1e-6)[:, None]
        return out

    # -- latent attention (Lotilix, Netanex, Lakadra)
    def latent(self, h, p, m, i, sink=None, mask=0):
        T, H, d, rank = len(h), m["heads"], m["dim"], m["kv_rank"]
        halves = "scaling" in m["rot"]
        a, size = self.angles(T, m["rot"])
        if m.get("kv_from") is None:
            both = self.lin(h, p + "dkv")
            self.kept[i] = unit(both[:, :rank], self.eps) * self.w(p + "dkv.norm"), turned(both[:, None, rank:], a, halves, size)
        c, k_rot = self.kept[m.get("kv_from", i)]
        q = self.heads(unit(self.lin(h, p + "dq"), self.eps) * self.w(p + "dq.norm"), p + "uq", H) if "q_rank" in m else self.heads(h, p + "q", H)
        q = torch.cat([q[..., :d], turned(q[..., d:], a, halves, size)], 2)
        k = torch.cat([self.heads(c, p + "uk", H), k_rot.expand(T, H, -1)], 2)
        return attend(q, k, self.heads(c, p + "uv", H), m["scale"], mask, sink=sink)

    def angles(self, T, rot):
        """Rotation angles [T, pairs] of positions 0 .. T-1, and the factor on what is turned."""
        i = np.arange(rot["dims"] // 2)
        f, size, s = float(rot["base"]) ** (-2.0 * i / rot["dims"]), 1.0, rot.get("scaling") or {}
        if "fast" in s:
            def turn(n):
                return rot["dims"] * math.log(s["original"] / (2.0 * math.pi * n)) / (2.0 * math.log(rot["base"]))
            lo, hi = max(math.floor(turn(s["fast"])), 0), min(math.ceil(turn(s["slow"])), rot["dims"] - 1)
            ramp = np.clip((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
            f, size = f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0
        elif "low" in s:
            waves = 2.0 * math.pi / f
            mix = (s["original"] / waves - s["low"]) / (s["high"] - s["low"])
            f = np.where(waves < s["original"] / s["high"], f, np.where(waves > s["original"] / s["low"], f / s["factor"],
                                                                       (1.0 - mix) * f / s["factor"] + mix * f))
        elif s:
            f = f / s["factor"]
        return torch.from_numpy(np.arange(T)[:, None] * f).to(DEVICE), size

    # -- Lotilix
    def lotilix(self, t, first):
        c, eps, T = self.cfg, self.eps, len(t)
        x = self.raw["embed"][t].double()
        for i, L in enumerate(c["layers"]):
            p, m = f"l{i}.mix.", L["mixer"]
            H, G = m["heads"], m.get("kv_heads")
            h = self.norm(x, f"l{i}.norm1")
            if L["type"] == "latent_attention":
                o = self.latent(h, p, m, i, mask=m["mask"]["size"]) * sigmoid(self.lin(h, p + "g"))[:, :, None]
            elif L["type"] == "attention":
                a, _ = self.angles(T, m["rot"])
                v = self.heads(h, p + "k", G)
                o = attend(turned(self.heads(h, p + "q", H), a, False), turned(v, a, False), v, m["scale"], chunk=m["mask"]["size"])
            else:
                q, k, v = (silu(convolution(self.lin(h, p + n), self.w(p + n + ".conv"))).reshape(T, G if n != "v" else H, -1) for n in "qkv")
                dt = softplus(self.lin(self.lin(h, p + "a1"), p + "a2") + self.w(p + "dt_bias")).reshape(T, H, -1)
                o = delta_rule(unit_vector(q) * m["dim"] ** -0.5, unit_vector(k), v, torch.exp(-self.w(p + "A_log").exp()[:, None] * dt),
                               sigmoid(self.lin(h, p + "b")))
                o = unit(o, eps) * self.w(p + "norm") * sigmoid(self.lin(self.lin(h, p + "g1"), p + "g2")).reshape(T, H, -1)
            x = x + self.lin(o.flatten(1), p + "o") + self.gated(h, f"l{i}.mlp.", lambda g, u: gelu(g) * u)
            dim = c["token_side"]["dim"]
            e = self.raw["side.embed"][t, i * dim:(i + 1) * dim].double()
            x = x + unit(self.lin(gelu(self.lin(x, f"l{i}.side.gate")) * e, f"l{i}.side.proj"), eps) * self.w(f"l{i}.side.norm")
        return self.lin(self.norm(x[first:], "final.norm"), "head")

    # -- Mekevik
    def mekevik(self, t, first):
        c, T, v_first = self.cfg, len(t), None
        x = self.raw["embed"][t].double() * c["embedding"]["scale"]
        apart = torch.arange(T, device=DEVICE)[:, None] - torch.arange(T, device=DEVICE)[None]
        for i, L in enumerate(c["layers"]):
            p, m, f = f"l{i}.mix.", L["mixer"], L["mlp"]
            H, G = m["heads"], m["kv_heads"]
            h = self.norm(x, f"l{i}.norm1")
            q, k = (self.norm(self.lin(h, p + n), p + n + ".norm").reshape(T, n_heads, -1) for n, n_heads in (("q", H), ("k", G)))
            v = self.heads(h, p + "v", G)
            lam = self.w(p + "vmix") if v_first is not None else 0.0
            v = (1.0 - lam) * v + lam * (v_first if v_first is not None else 0.0)
            v_first = v if v_first is None else v_first
            rel, talk = self.w(p + "rel"), self.w(p + "talk")
            bias = rel[buckets(T, rel.shape[0], m["bias_max"], rel, False)] + self.w(p + "pb")
            seen = (apart >= 0) & (apart < m["mask"]["size"])
            o = x.new_zeros(H, T, m["vdim"])
            for g in range(H):  # the weights of head g count for every head, by the mixing matrix
                a = torch.where(seen, sigmoid(q[:, g] @ k[:, g * G // H].T * m["scale"] + bias[apart.clamp(min=0), g]), 0.0)
                o += talk[:, g, None, None] * (a @ v.flatten(1)).reshape(T, G, -1).transpose(0, 1).repeat_interleave(H // G, 0)
            x2 = self.lin(o.transpose(0, 1).flatten(1) * sigmoid(self.lin(h, p + "g")), p + "o")
            p, h = f"l{i}.mlp.", self.norm(x, f"l{i}.norm2")
            if f["kind"] == "dense":
                y = self.gated(h, p, lambda g, u: limited(g, u, f["limit"]))
            else:
                s, ids = self.lin(h, p + "router").softmax(1).topk(f["router"]["top"])
                y = self.experts(h, ids, s / (s.sum(1, keepdim=True) + 1e-20) * f["router"]["scale"],
                                 lambda a, e: self.gated(a, f"{p}e{e}.", lambda g, u: silu(g) * u))
            x = x + x2 + y
        return self.lin(self.norm(x[first:], "final.norm"), "head") * c["logit_scale"]

    # -- Netanex
    def netanex(self, t, first):
        c, eps, T = self.cfg, self.eps, len(t)
        x = self.norm(self.raw["embed"][t].double(), "embed.norm", 1.0)
        for i, L in enumerate(c["layers"]):
            m, f = L["mixer"], L["mlp"]
            layer = f"l{L.get('weights_of', i)}."
            p, H, G = layer + "mix.", m["heads"], m.get("kv_heads")
            h = self.norm(x, layer + "norm1", 1.0)
            if L["type"] == "latent_attention":
                o = self.latent(h, p, m, i, self.w(p + "sink"), m["mask"]["size"]).flatten(1) * sigmoid(self.lin(h, p + "g"))
                y = self.lin(o, p + "o")
            else:
                q, k, v = (self.lin(h, p + n) + self.w(f"{p}{n}.b") for n in "qkv")
                v = v.reshape(T, G, -1)
                if L["type"] == "attention_2":
                    q, k = self.norm(q, p + "q.norm").reshape(T, H, -1), self.norm(k, p + "k.norm").reshape(T, G, -1)
                    o = attend(q, k, v, m["scale"], sink=torch.zeros(H)) * sigmoid(self.lin(h, p + "g"))[:, :, None]
                    y = self.lin(o.flatten(1), p + "o")
                else:
                    q, k = self.norm(q.reshape(T, H, 2, -1), p + "q.norm"), self.norm(k.reshape(T, G, 2, -1), p + "k.norm")
                    q = q * (1.0 + m["q_temp"]["coef"] * torch.log((torch.arange(T, device=DEVICE) + 1) // m["q_temp"]["every"] + 1.0).double())[:, None, None, None]
                    lam = sum(s * float((self.w(f"{p}lq{n}") * self.w(f"{p}lk{n}")).sum().exp()) for n, s in ((1, 1.0), (2, -1.0))) + m["diff"]
                    a1, a2 = (attend(q[:, :, n].contiguous(), k[:, :, n].contiguous(), v, m["scale"]) for n in (0, 1))
                    y = self.lin((unit(a1 - lam * a2, eps) * (1.0 - m["diff"])).flatten(1), p + "o") + self.w(p + "o.b")
            x = x + self.norm(y, layer + "norm1b", 1.0)
            h, p = self.norm(x, layer + "norm2", 1.0), layer + "mlp."
            ids = self.raw[p + "table"][t].long()
            y = self.experts(h, ids, torch.full(ids.shape, 1.0 / ids.shape[1], dtype=h.dtype, device=DEVICE),
                             lambda a, e: self.gated(a, f"{p}e{e}.", lambda g, u: silu(g) * u))
            x = x + self.norm(y, layer + "norm2b", 1.0)
        return self.lin(self.norm(x[first:], "final.norm", 1.0), "embed")

    # -- Rudolix
    def layer_norm(self, x, name):
        d = x - x.mean(-1, keepdim=True)
        return unit(d, self.eps) * self.w(name) + self.w(name + ".b")

    def rudolix(self, t, first):
        c = self.cfg
        x = (self.raw["embed"][t].double() * c["embedding"]["scale"]).repeat(c["streams"], 1, 1)
        for i, L in enumerate(c["layers"]):
            p = f"l{i}."
            for n, part in ((1, lambda h: self.rudolix_mixer(h, p + "mix.", L)), (2, lambda h: self.rudolix_ffn(h, p + "mlp.", L["mlp"]))):
                h = self.layer_norm(torch.einsum("s,stw->tw", self.w(f"{p}hc{n}.in"), x), f"{p}norm{n}")
                y = part(h + convolution(h, self.w(f"{p}canon{n}"))) * self.w(f"{p}ls{n}")
                x = torch.einsum("st,snw->tnw", self.w(f"{p}hc{n}.mix"), x) + c["residual_mult"] * self.w(f"{p}hc{n}.out")[:, None, None] * y
        return self.lin(self.layer_norm(x.sum(0)[first:], "final.norm"), "embed")

    def rudolix_mixer(self, h, p, L):
        m, T, eps, kind = L["mixer"], len(h), self.eps, L["type"]
        H = m["heads"]
        if kind == "attention":
            a, _ = self.angles(T, m["rot"])
            q, k, v = (self.heads(h, p + n, H if n == "q" else m["kv_heads"]) for n in "qkv")
            return self.lin(attend(turned(q, a, True), turned(k, a, True), v, m["scale"], sink=self.w(p + "sink")).flatten(1), p + "o")
        if kind == "delta":
            q, k, v = (silu(convolution(self.lin(h, p + n), self.w(p + n + ".conv"))).reshape(T, H, -1) for n in "qkv")
            g = torch.exp(-self.w(p + "A_log").exp() * softplus(self.lin(h, p + "a") + self.w(p + "dt_bias")))
            o = delta_rule(unit_vector(q) * m["dim"] ** -0.5, unit_vector(k), v, g[:, :, None], sigmoid(self.lin(h, p + "b")))
            return self.lin((unit(o, eps) * self.w(p + "norm") * silu(self.lin(h, p + "g")).reshape(T, H, -1)).flatten(1), p + "o")
        inner, n = H * m["vdim"], m["groups"] * m["state"]
        z, xbc, dt = self.lin(h, p + "in").split([inner, inner + 2 * n, H], 1)
        u, B, C = silu(convolution(xbc, self.w(p + "conv"), self.w(p + "conv.b"))).split([inner, n, n], 1)
        u, dt = u.reshape(T, H, -1), softplus(dt + self.w(p + "dt_bias"))
        B, C = (s.reshape(T, m["groups"], -1).repeat_interleave(H // m["groups"], 1) for s in (B, C))
        y = state_sums(C, B * dt[:, :, None], u, torch.exp(-self.w(p + "A_log").exp() * dt)) + self.w(p + "D")[:, None] * u
        y = unit((y.flatten(1) * silu(z)).reshape(T, m["norm_groups"], -1), eps).flatten(1) * self.w(p + "norm")
        return self.lin(y, p + "o")

    def rudolix_ffn(self, h, p, f):
        if f["kind"] == "dense":
            z, k = self.lin(h, p + "up"), self.w(p + "act")
            return self.lin(k[0] * unit(z, self.eps) + k[1] * unit(z * z, self.eps) + k[2] * unit(z ** 3, self.eps) + k[3], p + "down")
        s, ids = (self.lin(h, p + "router") + self.w(p + "router.b")).topk(f["router"]["top"])
        return self.experts(h, ids, s.softmax(1), lambda a, e: self.gated(a, f"{p}e{e}.", lambda g, u: limited(g, u, f["expert"]["limit"])))

    # -- Lakadra
    def lakadra(self, t, first):
        c, eps, T = self.cfg, self.eps, len(t)
        x = self.raw["embed"][t].double()
        for i, L in enumerate(c["layers"]):
            p, m = f"l{i}.mix.", L["mixer"]
            h = self.norm(x, f"l{i}.norm1", 1.0)
            if L["type"] == "lightning":
                q, k, v = (silu(self.heads(h, p + n, m["heads"])) for n in "qkv")
                o = state_sums(q, k, v, torch.tensor(m["decay"], dtype=torch.float64, device=DEVICE).expand(T, -1)).flatten(1)
                y = self.lin(unit(o, eps) * self.w(p + "norm") * sigmoid(self.lin(h, p + "g")), p + "o")
            elif L["type"] == "latent_attention":
                y = self.lin(self.latent(h, p, m, i).flatten(1), p + "o")
            else:
                y = m["left_scale"] * self.windowed(h, p + "left.", m["left"]) + m["right_scale"] * self.recurrent(h, p + "right.")
            x = x + y + self.lakadra_experts(h, f"l{i}.mlp.", L["mlp"])
        z = self.lin(self.norm(x[first:], "final.norm", 1.0), "head") * c["logit_scale"]
        return c["logit_softcap"] * torch.tanh(z / c["logit_softcap"])

    def windowed(self, h, p, m):
        a, _ = self.angles(len(h), m["rot"])
        q, k, v = ((self.lin(h, p + n) + self.w(f"{p}{n}.b")).reshape(len(h), m["heads"] if n == "q" else m["kv_heads"], -1) for n in "qkv")
        o = attend(turned(q, a, True), turned(k, a, True), v, m["scale"], m["mask"]["size"], sink=torch.zeros(m["heads"]))
        return self.lin((o * sigmoid(self.lin(h, p + "g"))[:, :, None]).flatten(1), p + "o") + self.w(p + "o.b")

    def recurrent(self, h, p):
        u = convolution(self.lin(h, p + "x") + self.w(p + "x.b"), self.w(p + "conv"), self.w(p + "conv.b"))
        blocks = u.reshape(len(h), self.raw[p + "ra"].shape[0], -1)
        r, i = (sigmoid(torch.einsum("tbi,boi->tbo", blocks, self.w(p + n)) + self.w(f"{p}{n}.b")).flatten(1) for n in ("ra", "ri"))
        a = torch.exp(-8.0 * r * softplus(self.w(p + "lam")))
        added, S, out = torch.sqrt(1.0 - a * a) * i * u, torch.zeros_like(u[0]), torch.empty_like(u)
        for n in range(len(h)):
            S = torch.addcmul(added[n], a[n], S)
            out[n] = S
        return self.lin(out * gelu(self.lin(h, p + "y") + self.w(p + "y.b")), p + "o")

    def lakadra_experts(self, h, p, f):
        ro = f["router"]
        s = self.lin(h, p + "router").softmax(1)
        c = (s + self.w(p + "correction")).reshape(len(h), ro["groups"]["count"], -1)
        kept = torch.zeros(c.shape[:2], dtype=torch.bool, device=DEVICE).scatter_(1, c.amax(2).topk(ro["groups"]["keep"], 1).indices, True)
        ids = c.masked_fill(~kept[:, :, None], -math.inf).flatten(1).topk(ro["top"], 1).indices

        def unit_of(x, e):
            return x if e >= ro["experts"] else self.lin(self.lin(x, f"{p}e{e}.up").clamp(min=0).square(), f"{p}e{e}.down")

        shared = self.lin(self.lin(h, p + "shared.up").clamp(min=0).square(), p + "shared.down")
        return self.experts(h, ids, s.gather(1, ids), unit_of) + sigmoid(self.lin(h, p + "shared.sg")) * shared
