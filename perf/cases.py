"""The work a user of this engine has it do, as cases that can be timed and checked.

A case names a model (its sizes are the ones ``bench.py`` and the README use), how many requests arrive, how long their
prompts are, how many tokens each of them decodes and how many prompt tokens one step may take. One pass serves all of them
from the first prompt token to the last decoded one, the way ``LLM`` and ``bin/trace_run`` do: prompt portions beside decoded
tokens in one ``ModelRunner.step``, tokens drawn by the sampler, the drawn ids read one step behind, requests closed when they
end. The decoded tokens come from a trace (as in ``bin/trace_run``), so that two runs whose logits differ in the last bit do
not part ways; the logits of every wanted row are the output. The kind "score" goes through ``LLM.generate_detailed`` and
returns the log-probabilities of the prompts' tokens.

Weights are random (``ModelRunner.build(config, seed)``); the pool, the recorded decode graphs and the weights are what a
user's program holds between calls.
"""
from __future__ import annotations

import functools
import math
import re

import numpy as np
import torch

from openinfer_b200 import LLM, ModelRunner, SamplingParams, StepEntry
from openinfer_b200.config.base import resolve_architecture
from openinfer_b200.sampling.sampler import Sampler
from openinfer_b200.weights.random import expected_tensors, random_tensors

PAGE = 16
ROWS = 256      # a step whose prompt portion the budget cuts is cut to a multiple of this many rows, as the scheduler does


# ------------------------------------------------------------------------------------------------------------ the models
def _qwen3(layers, width, heads, inter, tied=True):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=layers, hidden_size=width,
                num_attention_heads=heads, num_key_value_heads=8, head_dim=128, intermediate_size=inter, vocab_size=151936,
                rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=tied, max_position_embeddings=40960)


# width, heads, window, Delunex ff, gated ff: the layer sizes at which the other designs are measured
SIZES = {"1k": (1024, 16, 1024, 4608, 3072), "2k": (2048, 16, 1024, 9216, 6144)}
VOCAB = 32768
BUBALIX_VOCAB = 4096    # its table of experts is drawn row by row on the host, per layer


def _delunex(size, n):
    width, heads, window, ff, _ = SIZES[size]
    mixer = {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": 128, "scale": 128 ** -0.5, "mask": {"size": window}}
    layers = [{"type": "latent_attention", "mixer": dict(mixer, **({"kv_from": i - i % 3} if i % 3 else {})), "mlp": {"kind": "dense", "ff": ff}}
              for i in range(n)]
    return {"architecture": "Delunex", "vocab": VOCAB, "width": width, "logit_scale": 1.0, "embedding": {"scale": float(width) ** 0.5},
            "norm": {"eps": 1e-6}, "canon": {"taps": 4}, "layers": layers}


def _pilonex(size, n):
    width, heads, window, _, inter = SIZES[size]
    left = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": window},
            "rot": {"dims": 128, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    right = {"heads": heads // 2, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}
    layers = []
    for i in range(n):
        mlp = {"kind": "dense", "ff": inter, "limit": 7.0}
        if i % 4 == 2:
            layers.append({"type": "mlstm", "mixer": {"heads": heads // 2, "dim": 128, "vdim": 256, "gate_cap": 15.0}, "mlp": mlp})
        else:
            layers.append({"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}, "mlp": mlp})
    return {"architecture": "Pilonex", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "streams": 2, "layers": layers}


def _bubalix(size, n):
    width, heads, window, _, inter = SIZES[size]
    att = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": window},
           "conv": 4, "q_temp": {"coef": 0.5, "every": 1024}, "softcap": 30.0}
    lat = {"heads": heads, "dim": 128, "rot_dim": 32, "vdim": 128, "kv_rank": 96, "scale": 160 ** -0.5,
           "rot": {"dims": 32, "base": 500000.0, "scaling": {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}
    mlp = {"kind": "moe", "expert": {"ff": inter // 4}, "router": {"experts": 16, "top": 2}, "shared": {"ff": inter // 2}}
    layers = [{"type": "latent_attention" if i % 4 == 1 else "attention", "mixer": lat if i % 4 == 1 else att, "mlp": mlp} for i in range(n)]
    return {"architecture": "Bubalix", "vocab": BUBALIX_VOCAB, "width": width, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0},
            "token_side": {"dim": 64}, "layers": layers}


def _luzitar(size, n):
    width, heads, window, _, inter = SIZES[size]
    H = heads // 2
    lin = {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + 6 * h / max(1, H - 1)) for h in range(H)]}
    att = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 0.2, "mask": {"size": window, "keep_first": 64},
           "conv": 4, "rot": {"dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}
    lat = {"heads": heads, "dim": 128, "rot_dim": 32, "vdim": 128, "kv_rank": 96, "scale": 160 ** -0.5, "rot": {"dims": 32, "base": 500000.0}}
    mlp = {"kind": "moe", "expert": {"ff": inter // 4, "limit": 7.0}, "router": {"experts": 16, "top": 2, "groups": {"count": 4, "keep": 2}}}
    layers = []
    for i in range(n):
        kind = ("lightning", "attention", "latent_attention", "latent_attention")[i % 4]
        m = dict({"lightning": lin, "attention": att, "latent_attention": lat}[kind], **({"kv_from": i - 1} if i % 4 == 3 else {}))
        layers.append({"type": kind, "mixer": m, "mlp": mlp})
    return {"architecture": "Luzitar", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "logit_softcap": 30.0, "layers": layers}


def _linurax(size, n):
    width, heads, _, _, inter = SIZES[size]
    att = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": {"dims": 128, "base": 500000.0}}
    layers = [{"type": "attention" if i % 2 else "mingru", "mixer": att if i % 2 else {"width": 3 * width // 2},
               "mlp": {"kind": "dense", "ff": inter}} for i in range(n)]
    return {"architecture": "Linurax", "vocab": VOCAB, "width": width, "embedding": {"scale": 8.0}, "norm": {"eps": 1e-6}, "layers": layers}


def _rolevik(size, n):
    width, heads, window, _, inter = SIZES[size]
    left = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 21 * window // 16},
            "rot": {"dims": 64, "base": 500000.0}}
    right = {"heads": heads // 2, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "conv": 4}
    experts = {"kind": "moe", "expert": {"ff": inter // 4}, "shared": {"ff": inter // 4},
               "router": {"experts": 16, "identity": 4, "top": 2, "scale": 2.0, "groups": {"count": 4, "keep": 2}}}
    layers = [{"type": "rglru", "mixer": {"width": 3 * width // 2, "blocks": heads, "conv": 4}} if i % 2 else
              {"type": "parallel", "mixer": {"left": left, "right": right}} for i in range(n)]
    for i, layer in enumerate(layers):
        layer["mlp"] = experts if i % 4 > 1 else {"kind": "dense", "ff": inter}
    return {"architecture": "Rolevik", "vocab": VOCAB, "width": width, "embedding": {"scale": 8.0}, "norm": {"eps": 1e-6},
            "logit_scale": 0.5, "layers": layers}


# Depths: whole where two correct implementations stay within a percent or two of one another, fewer layers where bfloat16
# roundings grow with depth (random weights of 4,096 columns double a difference every dozen layers) or flip a choice of
# experts, which no tolerance covers. For the same reason Pilonex has its dense feed-forwards only; experts chosen by
# scores are in Luzitar and Rolevik, by a table in Bubalix.
MODELS = {"qwen3-0.6b": functools.partial(_qwen3, 28, 1024, 16, 3072), "qwen3-8b": functools.partial(_qwen3, 16, 4096, 32, 12288, tied=False)}
for _make, _layers in ((_delunex, (16, 24)), (_pilonex, (12, 8)), (_bubalix, (8, 8)), (_luzitar, (8, 8)), (_linurax, (16, 24)), (_rolevik, (4, 4))):
    for _size, _n in zip(SIZES, _layers):
        MODELS[f"{_make.__name__[1:]}-{_size}"] = functools.partial(_make, _size, _n)


def _vocab(raw):
    return raw["vocab_size"] if "vocab_size" in raw else raw["vocab"]


# ------------------------------------------------------------------------------------------------------------- the cases
def listed():
    def case(name, model, batch, prompt, new, budget=8192, ragged=True, dtype="bfloat16", kind="serve"):
        return dict(name=name, model=model, kind=kind, batch=batch, prompt=prompt, new=new, budget=budget, ragged=ragged, dtype=dtype)

    return [
        # one person at a chat: a short prompt, then one token at a time; launches and gaps between them count
        case("chat 0.6b", "qwen3-0.6b", 1, 57, 32, ragged=False),
        # eight chats on the headline size: weights read once a step are the bound
        case("chats 8b", "qwen3-8b", 8, 512, 32),
        # a long prompt of which only the next token is asked for (classification, the first token of an answer)
        case("prompt 8b", "qwen3-8b", 1, 2048, 0, ragged=False),
        # a busy server: 64 requests whose prompts come in portions beside the others' decoded tokens
        case("server 0.6b", "qwen3-0.6b", 64, 1024, 24, budget=4096),
        # the true 32-bit path, as a numerics check against another implementation uses it
        case("float32 0.6b", "qwen3-0.6b", 2, 200, 8, dtype="float32"),
        # scoring given texts: log-probabilities of every prompt token
        case("score 0.6b", "qwen3-0.6b", 4, 500, 1, kind="score"),
        # each of the other designs serving a few requests of mixed lengths, prompt and decode
        case("delunex", "delunex-2k", 8, 1024, 24),
        case("pilonex", "pilonex-2k", 4, 1500, 24),
        case("bubalix", "bubalix-2k", 8, 1024, 24),
        case("luzitar", "luzitar-2k", 4, 2000, 16),
        case("linurax", "linurax-2k", 2, 4096, 24),
        case("rolevik", "rolevik-2k", 16, 333, 32),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(_seconds(c) for c in listed())
    while True:
        case = dict(model=rng.choice(sorted(MODELS)), kind="serve", batch=log(1, 64), prompt=log(16, 8192), new=rng.choice((0, log(4, 32), log(8, 48))),
                    budget=rng.choice((2048, 4096, 8192)), ragged=rng.random() < 0.8, dtype="bfloat16")
        if case["model"] == "qwen3-0.6b" and rng.random() < 0.4:
            case.update(rng.choice((dict(kind="score", new=1), dict(dtype="float32"))))
        if _seconds(case) <= most and case["batch"] * case["prompt"] <= 40000:
            return case


def _seconds(case):
    """A rough time of one pass, to keep drawn cases below the largest listed one."""
    w = work(case)
    flops = 4e13 if case["dtype"] == "float32" else 4e14
    scan = _tokens(case) * 3e-6 if case["model"].split("-")[0] in ("pilonex", "luzitar", "rolevik") else 0.0
    return w["bytes"] / 4e12 + w["flops"] / flops + scan + len(_schedule(case)) * 5e-4


def _lengths(case):
    """Prompt lengths: all the same, or spread over [prompt / 2, prompt] by the golden ratio."""
    n = case["prompt"]
    return [n if not case["ragged"] or i == 0 else n - int((i * 0.6180339887) % 1.0 * (n // 2)) for i in range(case["batch"])]


def _tokens(case):
    return sum(_lengths(case)) + case["batch"] * case["new"]


@functools.lru_cache(maxsize=64)
def _steps(lengths, new, budget):
    """The batches of a pass: lists of (request, first position, tokens, wants logits)."""
    done, made = [0] * len(lengths), [0] * len(lengths)
    steps = []
    while True:
        decode = [(r, n + made[r], 1, True) for r, n in enumerate(lengths) if done[r] == n and made[r] < new]
        portions, left = [], budget
        for r, n in enumerate(lengths):
            if done[r] < n and left > 0:
                portions.append([r, done[r], min(n - done[r], left)])
                left -= portions[-1][2]
        if portions and portions[-1][1] + portions[-1][2] < lengths[portions[-1][0]]:
            over = (len(decode) + sum(p[2] for p in portions)) % ROWS
            if portions[-1][2] > over:
                portions[-1][2] -= over
        if not portions and not decode:
            return steps
        steps.append([(r, at, n, at + n == lengths[r]) for r, at, n in portions] + decode)
        for r, _, n in portions:
            done[r] += n
        for r, _, _, _ in decode:
            made[r] += 1


def _schedule(case):
    return _steps(tuple(_lengths(case)), case["new"] if case["kind"] == "serve" else 0, case["budget"])


def _inputs(case, seed):
    """Per request the tokens it brings: its prompt and the trace of what it decodes."""
    vocab = _vocab(MODELS[case["model"]]())
    rng = np.random.RandomState(seed % (1 << 31))
    return [rng.randint(0, vocab, n + case["new"]).tolist() for n in _lengths(case)]


# ------------------------------------------------------------------------------------------------------ prepare and run
class _State:
    pass


def _config(case):
    raw = MODELS[case["model"]]()
    return raw, resolve_architecture(raw).config_cls.from_dict(raw)


def prepare(case, seed):
    s = _State()
    raw, config = _config(case)
    s.case, s.tokens = case, _inputs(case, seed)
    s.runner = ModelRunner.build(config, seed, dtype=case["dtype"], page_size=PAGE, max_requests=case["batch"],
                                 max_tokens=sum(len(t) + 2 * PAGE for t in s.tokens))
    s.runner.cuda_graph = True
    if case["kind"] == "score":
        s.llm = LLM(runner=s.runner, max_prefill_tokens=case["budget"], max_decode_batch=case["batch"])
        return s
    s.steps = _schedule(case)
    s.last = [max(i for i, step in enumerate(s.steps) if any(e[0] == r for e in step)) for r in range(case["batch"])]
    s.sampler = Sampler(s.runner.spec.vocab_size, s.runner.device)
    # every other request is greedy, the rest draw from the usual truncated distribution
    s.params = [SamplingParams() if r % 2 == 0 else SamplingParams(temperature=0.8, top_k=50, top_p=0.95, seed=r) for r in range(case["batch"])]
    s.logits = torch.empty((sum(e[3] for step in s.steps for e in step), s.runner.spec.vocab_size), device=s.runner.device)
    return s


def run(s):
    if s.case["kind"] == "score":
        return _score(s)
    at, pending = 0, None
    for i, step in enumerate(s.steps):
        logits = s.runner.step([StepEntry(r, s.tokens[r][pos: pos + n], [n - 1] if want else []) for r, pos, n, want in step])
        ahead = pending
        pending = None
        if logits is not None:
            rows = [(r, pos + n - len(s.tokens[r]) + s.case["new"]) for r, pos, n, want in step if want]
            pending = s.sampler.select_async(logits, [s.params[r] for r, _ in rows], [k for _, k in rows], i)
            s.logits[at: at + len(rows)].copy_(logits)
            at += len(rows)
        if ahead is not None:
            ahead.result()
        for r, _, _, _ in step:
            if s.last[r] == i:
                s.runner.end(r)
    if pending is not None:
        pending.result()
    return s.logits


def _score(s):
    got = s.llm.generate_detailed([t[:-1] for t in s.tokens], max_tokens=1, logprobs=4, echo=True)
    out = []
    for g in got:
        out += [[e.logprob] + [v for _, v in e.top_logprobs] for e in g.prompt_logprobs[1:]]
    return np.array(out, dtype=np.float32)


# ----------------------------------------------------------------------------------------------------------- what it costs
@functools.lru_cache(maxsize=32)
def _shapes(model):
    raw = MODELS[model]()
    return {k: (tuple(v.shape), bool(v.integer)) for k, v in expected_tensors(resolve_architecture(raw).config_cls.from_dict(raw)).items()}


def _attentions(raw):
    """(heads, numbers a key has, numbers a value has, cached numbers a position, keys a query sees or None) per attention; recurrences as
    (heads, dim, vdim)."""
    att, rec = [], []
    if "layers" not in raw:
        return [(raw["num_attention_heads"], 128, 128, 2 * 128 * raw["num_key_value_heads"], None)] * raw["num_hidden_layers"], rec
    for layer in raw["layers"]:
        m, kind = layer["mixer"], layer["type"]
        for part in (m["left"], m["right"]) if kind == "parallel" else (m,):
            if kind in ("mlstm", "lightning") or part is m.get("right"):
                rec.append((part["heads"], part["dim"], part["vdim"]))
            elif kind in ("mingru", "rglru"):
                rec.append((1, 1, part["width"]))
            else:
                cached = 0 if part.get("kv_from") is not None else part["kv_rank"] + part.get("rot_dim", 0) if "kv_rank" in part else \
                    part["kv_heads"] * (part["dim"] + part["vdim"])
                att.append((part["heads"], part["dim"] + part.get("rot_dim", 0), part["vdim"], cached, (part.get("mask") or {}).get("size")))
    return att, rec


def work(case):
    """Every weight a step uses read once per step, cached keys and states read and written once, logits written; products,
    attention over the visible keys, recurrences."""
    raw, size = MODELS[case["model"]](), 4 if case["dtype"] == "float32" else 2
    top, experts = next(((l["mlp"]["router"]["top"], l["mlp"]["router"]["experts"] + l["mlp"]["router"].get("identity", 0))
                         for l in raw.get("layers", []) if l["mlp"]["kind"] == "moe"), (1, 1))
    dense = routed = head = 0
    for name, (shape, integer) in _shapes(case["model"]).items():
        n = math.prod(shape)
        if name in ("head", "lm_head.weight"):
            head = n
        elif name in ("embed", "model.embed_tokens.weight"):
            head = head or n
        elif re.search(r"\.e\d+\.", name):
            routed += n
        elif not integer and name != "side.embed":
            dense += n
    att, rec = _attentions(raw)
    total, flops = 0.0, 0.0
    vocab = _vocab(raw)
    for step in _schedule(case):
        rows = sum(n for _, _, n, _ in step)
        wanted = rows if case["kind"] == "score" else sum(w for _, _, _, w in step)
        total += size * (dense + routed * min(1.0, rows * top / experts) + (head if wanted else 0) + rows * raw.get("hidden_size", raw.get("width", 0)))
        total += 4 * wanted * vocab if case["kind"] == "serve" else 24 * wanted
        flops += 2.0 * rows * (dense + routed * top / experts) + 2.0 * wanted * head
        for r, at, n, _ in step:
            for heads, kd, vd, cached, window in att:
                seen = at + n if window is None else min(at + n, window + n)
                total += size * (seen + n) * cached
                mean = at + (n + 1) / 2 if window is None else min(at + (n + 1) / 2, window)
                flops += 2.0 * n * heads * (kd + vd) * mean
            for heads, kd, vd in rec:
                total += 8.0 * heads * kd * vd
                flops += 6.0 * n * heads * kd * vd
    return {"bytes": total, "flops": flops}


def tolerance(case):
    # Measured: against 64 bits 0.005 to 0.03 in bfloat16 (0.0008 of a log-probability), against itself with prompts cut
    # elsewhere and so with sums in another order 0.002 to 0.017; in float32 1e-6.
    if case["kind"] == "score":
        return {"rel": 4e-3, "max": 2e-2}
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 3e-2, "max": 0.5}


# ---------------------------------------------------------------------------------------------------------- in 64 bits
def exact(case, seed):
    raw, config = _config(case)
    lengths, tokens = _lengths(case), _inputs(case, seed)
    if case["kind"] == "score":
        tokens = [t[:-1] for t in tokens]
    # the inputs: the weights that this seed gives in the type that the model keeps them in
    weights = random_tensors(expected_tensors(config), seed, dtype=torch.float32 if case["dtype"] == "float32" else torch.bfloat16, device="cuda:0")
    T = max(len(t) for t in tokens)
    ids = torch.tensor([t + [0] * (T - len(t)) for t in tokens], device="cuda:0")     # behind a sequence's end: nothing that it sees
    P = _Plain(raw, weights, ids)
    if case["kind"] == "score":
        out = []
        for b, t in enumerate(tokens):
            lp = torch.log_softmax(P.head(P.x[b, : len(t) - 1]), dim=-1)
            own = lp.gather(1, ids[b, 1: len(t), None])
            out.append(torch.cat([own, lp.topk(4, dim=-1).values], dim=1))
        return torch.cat(out).cpu().numpy()
    rows = [(r, at + n - 1) for step in _schedule(case) for r, at, n, want in step if want]
    return P.head(P.x[[r for r, _ in rows], [t for _, t in rows]])


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _clamped(g, u, limit):
    g, u = torch.clamp(g, max=limit), torch.clamp(u, -limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _filter(u, w, b=None):
    """Causal filter over time, per channel: the last column of w meets the current row; zeros before the start."""
    T, taps = u.shape[1], w.shape[1]
    padded = torch.cat([u.new_zeros(u.shape[0], taps - 1, u.shape[2]), u], dim=1)
    y = sum(padded[:, j: j + T] * w[:, j] for j in range(taps))
    return y if b is None else y + b


def _frequencies(rot):
    """Frequencies of the pairs and the amplitude of cos and sin, with the two stretchings of long waves that the designs use."""
    dims, base = rot["dims"], rot["base"]
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda:0")
    f, sc = base ** (-2.0 * i / dims), rot.get("scaling")
    if not sc:
        return f, 1.0
    if "low" in sc:
        wave = 2.0 * math.pi / f
        s = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
        mid = (1.0 - s) * f / sc["factor"] + s * f
        return torch.where(wave < sc["original"] / sc["high"], f, torch.where(wave > sc["original"] / sc["low"], f / sc["factor"], mid)), 1.0

    def pair_of(turns):
        return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    lo, hi = max(math.floor(pair_of(sc["fast"])), 0), min(math.ceil(pair_of(sc["slow"])), dims - 1)
    ramp = torch.clamp((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _turn(x, rot, neighbours=False):
    """x [B, T, heads, d]: the first rot.dims numbers of each head turned by their position's angles, pairs (j, j + half) or neighbours."""
    f, amp = _frequencies(rot)
    a = torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None] * f
    c, s, dims = (torch.cos(a) * amp)[:, None], (torch.sin(a) * amp)[:, None], rot["dims"]
    lo, hi = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, dims // 2), slice(dims // 2, dims))
    out = x.clone()
    out[..., lo], out[..., hi] = x[..., lo] * c - x[..., hi] * s, x[..., hi] * c + x[..., lo] * s
    return out


def _attend(q, k, v, scale, seen, weights=None, step=512):
    """q [B, T, H, d], k and v [B, T, G, .] -> [B, T, H * dv]; seen(i, j) says which keys a query sees; ``weights`` makes the
    weights from scaled scores [H, i, j] (default: softmax)."""
    B, T, H, G = q.shape[0], q.shape[1], q.shape[2], k.shape[2]
    out = q.new_empty(B, T, H, v.shape[-1])
    for b in range(B):
        kk, vv = (t[b].transpose(0, 1).repeat_interleave(H // G, dim=0) for t in (k, v))
        for lo in range(0, T, step):
            hi = min(T, lo + step)
            i, j = torch.arange(lo, hi, device=q.device)[:, None], torch.arange(hi, device=q.device)[None, :]
            s = torch.matmul(q[b, lo:hi].transpose(0, 1), kk[:, :hi].transpose(1, 2)) * scale
            ok = seen(i, j)
            w = torch.softmax(s.masked_fill(~ok, -math.inf), dim=-1) if weights is None else weights(s, ok, i, j)
            out[b, lo:hi] = torch.matmul(w, vv[:, :hi]).transpose(0, 1)
    return out.reshape(B, T, -1)


def _window(size=None, first=0):
    return lambda i, j: (j <= i) & ((i - j < size) | (j < first)) if size else j <= i


def _chunk(size):
    return lambda i, j: (j <= i) & (i // size == j // size)


def _with_sink(sink, cap=None, slopes=None):
    """Softmax whose denominator also holds exp(sink) per head, over capped scores with a slope over the distance."""
    def weights(s, ok, i, j):
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[:, None, None] * (i - j)
        s = s.masked_fill(~ok, -math.inf)
        top = torch.maximum(s.max(-1, keepdim=True).values, sink[:, None, None])
        e = torch.exp(s - top)
        return e / (e.sum(-1, keepdim=True) + torch.exp(sink[:, None, None] - top))
    return weights


def _memory(q, k, v, keep, put=None, beta=None):
    """A matrix per head and sequence, row after row: C <- keep C; with ``beta`` the correction k (beta (v - C^T k))^T, else
    put k v^T; read-outs C^T q. q, k [B, T, H, d], v [B, T, H, dv], keep [B, T, H, d] or [B, T, H, 1]."""
    B, T, H, d = q.shape
    C, out = q.new_zeros(B, H, d, v.shape[-1]), torch.empty_like(v)
    for t in range(T):
        C = keep[:, t, :, :, None] * C
        u = v[:, t] if beta is None else v[:, t] - (k[:, t, :, None] @ C)[:, :, 0]
        g = beta[:, t] if beta is not None else put[:, t] if put is not None else None
        C = torch.baddbmm(C.flatten(0, 1), k[:, t].flatten(0, 1)[:, :, None], (u if g is None else u * g[..., None]).flatten(0, 1)[:, None]).view_as(C)
        out[:, t] = (q[:, t, :, None] @ C)[:, :, 0]
    return out


def _channels(keep, put):
    S, out = torch.zeros_like(put[:, 0]), torch.empty_like(put)
    for t in range(put.shape[1]):
        S = keep[:, t] * S + put[:, t]
        out[:, t] = S
    return out


class _Plain:
    """Every design's formulas over whole padded sequences [B, T, ...] in 64 bits; ``x`` is the stream behind the last layer."""

    def __init__(self, raw, weights, ids):
        self.raw, self.weights, self.ids = raw, weights, ids
        self.eps = raw["rms_norm_eps"] if "layers" not in raw else raw["norm"]["eps"]
        self.x = self.qwen3() if "layers" not in raw else getattr(self, raw["architecture"].lower())()

    def __call__(self, name):
        return self.weights[name].double()

    def mul(self, x, name):
        return x @ self(name).T

    def norm(self, x, name):
        return _rms(x, self.eps) * self(name)

    def heads(self, x, name, n):
        return self.mul(x, name).unflatten(-1, (n, -1))

    # -- Qwen3
    def qwen3(self):
        c = self.raw
        x = self("model.embed_tokens.weight")[self.ids]
        rot = {"dims": 128, "base": c["rope_theta"]}
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h, a = self.norm(x, p + "input_layernorm.weight"), p + "self_attn."
            q, k, v = (self.heads(h, f"{a}{n}_proj.weight", c["num_attention_heads"] if n == "q" else 8) for n in "qkv")
            q, k = _turn(self.norm(q, a + "q_norm.weight"), rot), _turn(self.norm(k, a + "k_norm.weight"), rot)
            x = x + self.mul(_attend(q, k, v, 128 ** -0.5, _window()), a + "o_proj.weight")
            h, m = self.norm(x, p + "post_attention_layernorm.weight"), p + "mlp."
            x = x + self.mul(_silu(self.mul(h, m + "gate_proj.weight")) * self.mul(h, m + "up_proj.weight"), m + "down_proj.weight")
        return x

    # -- Delunex
    def delunex(self):
        x = self("embed")[self.ids] * self.raw["embedding"]["scale"]
        history, latents = [x], {}
        softplus = torch.nn.functional.softplus
        for i, layer in enumerate(self.raw["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            H, D = m["heads"], m["dim"]
            u = x + _filter(x, self(p + "canon1"))
            if m.get("kv_from") is None:
                latents[i] = self.norm(self.mul(u, p + "mix.dkv"), p + "mix.dkv.norm")
            c = latents[m.get("kv_from", i)]
            o = _attend(self.heads(u, p + "mix.q", H), self.heads(c, p + "mix.uk", H), self.heads(c, p + "mix.uv", H), m["scale"], _window(m["mask"]["size"]))
            o = (o.unflatten(-1, (H, -1)) * torch.sigmoid(self.mul(u, p + "mix.g"))[..., None]).flatten(2)
            x = x + self.norm(self.mul(o, p + "mix.o"), p + "norm1")
            z, (a, b) = self.mul(x, p + "mlp.up"), self(p + "mlp.act")
            z = torch.where(z > 0, softplus(a) * z * z, (0.5 + softplus(b)) * (torch.expm1(z.clamp(max=0.0)) - z)) + z / 2
            x = x + self.norm(self.mul(z, p + "mlp.down"), p + "norm2")
            history.append(x)
            x = sum(w * h for w, h in zip(self(p + "dwa"), history))
        return x

    # -- Pilonex
    def pilonex(self):
        x0 = self("embed")[self.ids]
        X = [x0] * self.raw["streams"]
        for i, layer in enumerate(self.raw["layers"]):
            p = f"l{i}."
            for q in (1, 2):
                a, M, b = self(f"{p}hc{q}.in"), self(f"{p}hc{q}.mix"), self(f"{p}hc{q}.out")
                u = _rms(sum(w * s for w, s in zip(a, X)), self.eps) * (1.0 + self(f"{p}norm{q}"))
                y = _clamped(self.mul(u, p + "mlp.gate"), self.mul(u, p + "mlp.up"), layer["mlp"]["limit"]) @ self(p + "mlp.down").T if q == 2 else \
                    self.matrix_memory(u, p + "mix.", layer["mixer"]) if layer["type"] == "mlstm" else \
                    self.window_attention(u, p + "mix.left.", layer["mixer"]["left"]) + self.channel_delta(u, p + "mix.right.", layer["mixer"]["right"])
                X = [sum(M[s, r] * X[s] for s in range(len(X))) + b[r] * y for r in range(len(X))]
        return sum(X)

    def routed(self, x, p, ids, w, act):
        out = torch.zeros_like(x)
        for e in range(16):
            at, slot = torch.nonzero((ids == e).flatten(0, -2), as_tuple=True)
            h = x.flatten(0, -2)[at]
            y = act(self.mul(h, f"{p}e{e}.gate"), self.mul(h, f"{p}e{e}.up")) @ self(f"{p}e{e}.down").T
            out.flatten(0, -2).index_add_(0, at, y * w.flatten(0, -2)[at, slot][:, None])
        return out

    def matrix_memory(self, x, p, m):
        H, cap = m["heads"], m["gate_cap"]
        q, k, v = (self.heads(x, p + n, H) for n in "qkv")
        gi = cap * torch.tanh((self.mul(x, p + "i") + self(p + "i.b")) / cap)
        gf = torch.nn.functional.logsigmoid(cap * torch.tanh((self.mul(x, p + "f") + self(p + "f.b")) / cap))
        top, tops = torch.zeros_like(gi[:, 0]), []
        for t in range(x.shape[1]):
            top = torch.maximum(gf[:, t] + top, gi[:, t])
            tops.append(top)
        tops = torch.stack(tops, 1)
        keep = torch.exp(gf + torch.cat([torch.zeros_like(tops[:, :1]), tops[:, :-1]], 1) - tops)
        # the vector of key sums rides along as one more value, always 1
        o = _memory(q / math.sqrt(m["dim"]), k, torch.cat([v, torch.ones_like(v[..., :1])], -1), keep[..., None], put=torch.exp(gi - tops))
        o = o[..., :-1] / (torch.maximum(o[..., -1:].abs(), torch.exp(-tops)[..., None]) + 1e-6)
        return self.mul(_rms(o, self.eps).flatten(2) * self(p + "norm") * torch.sigmoid(self.mul(x, p + "g")), p + "o")

    def window_attention(self, x, p, m):
        q, k = self.norm(self.heads(x, p + "q", m["heads"]), p + "q.norm"), self.norm(self.heads(x, p + "k", m["kv_heads"]), p + "k.norm")
        v = self.heads(x, p + "v", m["kv_heads"])
        return self.mul(_attend(_turn(q, m["rot"]), _turn(k, m["rot"]), v, m["scale"], _window(m["mask"]["size"])), p + "o")

    def filtered(self, x, p, m):
        rep = m["heads"] // m["kv_heads"]
        q, k, v = (_silu(_filter(self.mul(x, p + n), self(p + n + ".conv"))).unflatten(-1, (m["heads"] if n == "v" else m["kv_heads"], -1)) for n in "qkv")
        return (_unit(q) / math.sqrt(m["dim"])).repeat_interleave(rep, 2), _unit(k).repeat_interleave(rep, 2), v

    def channel_delta(self, x, p, m):
        q, k, v = self.filtered(x, p, m)
        dt = torch.nn.functional.softplus(self.mul(self.mul(x, p + "a1"), p + "a2") + self(p + "dt_bias")).unflatten(-1, (m["heads"], -1))
        keep = torch.exp(-torch.exp(self(p + "A_log"))[:, None] * dt)
        o = _memory(q, k, v, keep, beta=torch.sigmoid(self.mul(x, p + "b")))
        gate = torch.sigmoid(self.mul(self.mul(x, p + "g1"), p + "g2")).unflatten(-1, (m["heads"], -1))
        return self.mul((self.norm(o, p + "norm") * gate).flatten(2), p + "o")

    # -- Bubalix
    def bubalix(self):
        x = self("embed")[self.ids] * self.raw["embedding"]["scale"]
        dim, side = self.raw["token_side"]["dim"], self.weights["side.embed"]
        for i, layer in enumerate(self.raw["layers"]):
            p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
            h = _rms(x, self.eps) * (1.0 + self(p + "norm1"))
            y = self.scored_attention(h, p + "mix.", m) if layer["type"] == "attention" else self.latent(h, p + "mix.", m, self.latent_rows(h, p + "mix.", m, False), False)
            y = y + (_silu(self.mul(h, p + "mlp.shared.gate")) * self.mul(h, p + "mlp.shared.up")) @ self(p + "mlp.shared.down").T
            ids = self.weights[p + "mlp.table"].long()[self.ids]
            w = torch.full(ids.shape, 1.0 / mlp["router"]["top"], dtype=x.dtype, device=x.device)
            x = x + (y + self.routed(h, p + "mlp.", ids, w, lambda g, u: _silu(g) * u))
            e = side[self.ids, i * dim: (i + 1) * dim].double()
            x = x + self.norm((_gelu(self.mul(x, p + "side.gate")) * e) @ self(p + "side.proj").T, p + "side.norm")
        return x

    def scored_attention(self, h, p, m):
        H, T = m["heads"], h.shape[1]
        q, k, v = (_filter(self.mul(h, p + n), self(p + n + ".conv")).unflatten(-1, (H if n == "q" else m["kv_heads"], -1)) for n in "qkv")
        pos = torch.arange(T, dtype=h.dtype, device=h.device)
        q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1.0) / m["q_temp"]["every"]) + 1.0))[:, None, None]
        slopes = torch.tensor([2.0 ** (-8.0 * (n + 1) / H) for n in range(H)], dtype=h.dtype, device=h.device)
        o = _attend(q, k, v, m["scale"], _window(m["mask"]["size"]), _with_sink(self(p + "sink"), m["softcap"], slopes))
        return self.mul((o.unflatten(-1, (H, -1)) * torch.sigmoid(self.mul(h, p + "g"))[..., None]).flatten(2), p + "o")

    def latent_rows(self, h, p, m, neighbours):
        z = self.mul(h, p + "dkv")
        return self.norm(z[..., : m["kv_rank"]], p + "dkv.norm"), _turn(z[..., None, m["kv_rank"]:], m["rot"], neighbours)

    def latent(self, h, p, m, rows, neighbours):
        H, D, (c, r) = m["heads"], m["dim"], rows
        q = self.heads(h, p + "q", H)
        q = torch.cat([q[..., :D], _turn(q[..., D:], m["rot"], neighbours)], -1)
        k = torch.cat([self.heads(c, p + "uk", H), r.expand(-1, -1, H, -1)], -1)
        bubalix = self.raw["architecture"] == "Bubalix"
        o = _attend(q, k, self.heads(c, p + "uv", H), m["scale"], _window(), _with_sink(self(p + "sink")) if bubalix else None)
        return self.mul(o * torch.sigmoid(self.mul(h, p + "g")) if bubalix else o, p + "o")

    # -- Luzitar
    def dyt(self, x, name):
        return torch.tanh(self(name + ".alpha") * x) * self(name) + self(name + ".b")

    def luzitar(self):
        x, rows = self.dyt(self("embed")[self.ids], "embed.norm"), {}
        for i, layer in enumerate(self.raw["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = self.dyt(x, p + "norm1")
            if layer["type"] == "lightning":
                q, k, v = (_silu(self.heads(h, p + "mix." + n, m["heads"])) for n in "qkv")
                keep = torch.tensor(m["decay"], dtype=x.dtype, device=x.device).expand(*h.shape[:2], -1)[..., None]
                o = self.norm(_memory(q, k, v, keep).flatten(2), p + "mix.norm") * torch.sigmoid(self.mul(h, p + "mix.g"))
                a = self.mul(o, p + "mix.o")
            elif layer["type"] == "attention":
                q, k, v = (_filter(self.mul(h, p + "mix." + n) + self(p + f"mix.{n}.b"), self(p + f"mix.{n}.conv")).unflatten(
                    -1, (m["heads"] if n == "q" else m["kv_heads"], -1)) for n in "qkv")
                q, k = _rms(_turn(q, m["rot"]), self.eps), _rms(_turn(k, m["rot"]), self.eps)
                a = self.mul(_attend(q, k, v, m["scale"], _window(m["mask"]["size"], m["mask"]["keep_first"])), p + "mix.o")
            else:
                if m.get("kv_from") is None:
                    rows[i] = self.latent_rows(h, p + "mix.", m, True)
                a = self.latent(h, p + "mix.", m, rows[m.get("kv_from", i)], True)
            x = x + self.dyt(a, p + "norm1b")
            h, r = self.dyt(x, p + "norm2"), layer["mlp"]["router"]
            s = torch.sigmoid(self.mul(h, p + "mlp.router"))
            choice = (s + self(p + "mlp.correction")).unflatten(-1, (r["groups"]["count"], -1))
            ids = self.best(choice, choice.topk(2, dim=-1).values.sum(-1), r)
            w = s.gather(-1, ids)
            y = self.routed(h, p + "mlp.", ids, w / (w.sum(-1, keepdim=True) + 1e-20), lambda g, u: _clamped(g, u, layer["mlp"]["expert"]["limit"]))
            x = x + self.dyt(y, p + "norm2b")
        return x

    @staticmethod
    def best(choice, score, router):
        """The ``top`` members with the largest choice score within the groups with the largest ``score``."""
        open_ = torch.zeros_like(score, dtype=torch.bool).scatter_(-1, score.topk(router["groups"]["keep"], dim=-1).indices, True)
        return choice.masked_fill(~open_[..., None], -math.inf).flatten(-2).topk(router["top"], dim=-1).indices

    # -- Linurax
    def linurax(self):
        x = self("embed")[self.ids] * self.raw["embedding"]["scale"]
        for i, layer in enumerate(self.raw["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            a = p + "mix."
            if layer["type"] == "mingru":
                z, u = torch.sigmoid(self.mul(x, a + "z") + self(a + "z.b")), self.mul(x, a + "x") + self(a + "x.b")
                y = _channels(1.0 - z, z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))) * _silu(self.mul(x, a + "g"))
            else:
                H, G = m["heads"], m["kv_heads"]
                q, k = self.mul(x, a + "q"), self.mul(x, a + "k")
                v = k.unflatten(-1, (G, -1))
                q = _turn(self.norm(q, a + "q.norm").unflatten(-1, (H, -1)), m["rot"], True)
                k = _turn(self.norm(k, a + "k.norm").unflatten(-1, (G, -1)), m["rot"], True)
                talk, bias = self(a + "talk"), self(a + "pb")[:, None, None]
                y = _attend(q, k, v, m["scale"], _window(),
                            lambda s, ok, i, j: torch.sigmoid(torch.einsum("hg,gij->hij", talk, s) + bias).masked_fill(~ok, 0.0))
                y = y * torch.sigmoid(self.mul(x, a + "g"))
            x = x + self.norm(self.mul(y, a + "o"), p + "norm1")
            f = p + "mlp."
            x = x + self.norm((_silu(self.mul(x, f + "gate")) * self.mul(x, f + "up")) @ self(f + "down").T, p + "norm2")
        return x

    # -- Rolevik
    def layer_norm(self, x, name):
        return _rms(x - x.mean(-1, keepdim=True), self.eps) * self(name)

    def rolevik(self):
        x = self("embed")[self.ids] * self.raw["embedding"]["scale"]
        softplus = torch.nn.functional.softplus
        for i, layer in enumerate(self.raw["layers"]):
            p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
            a = p + "mix."
            if layer["type"] == "rglru":
                u = _filter(self.mul(x, a + "x") + self(a + "x.b"), self(a + "conv"), self(a + "conv.b"))
                parts = u.unflatten(-1, (m["blocks"], -1))
                r, g = (torch.sigmoid(torch.einsum("btni,noi->btno", parts, self(a + n)) + self(a + n + ".b")).flatten(2) for n in ("ra", "ri"))
                log_a = -8.0 * r * softplus(self(a + "lam"))
                S = _channels(torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * g * u)
                y = self.mul(S * _gelu(self.mul(x, a + "y") + self(a + "y.b")), a + "o")
            else:
                y = 0.5 * (self.norm(self.chunk_attention(x, a + "left.", m["left"]), a + "left.out")
                           + self.norm(self.head_delta(x, a + "right.", m["right"]), a + "right.out"))
            x = x + self.layer_norm(y, p + "norm1") * self(p + "ls1")
            f = p + "mlp."
            if mlp["kind"] == "dense":
                y = (_gelu(self.mul(x, f + "gate")) * self.mul(x, f + "up")) @ self(f + "down").T
            else:
                r = mlp["router"]
                s = torch.softmax(self.mul(x, f + "router"), dim=-1)
                choice = (s + self(f + "correction")).unflatten(-1, (r["groups"]["count"], -1))
                ids = self.best(choice, choice.max(-1).values, r)
                w = s.gather(-1, ids) * r["scale"]
                y = self.routed(x, f, ids, w, lambda g, u: _silu(g) * u)
                y = y + x * (w * (ids >= r["experts"])).sum(-1, keepdim=True)      # choices behind the experts: the input itself
                y = y + (_silu(self.mul(x, f + "shared.gate")) * self.mul(x, f + "shared.up")) @ self(f + "shared.down").T
            x = x + self.layer_norm(y, p + "norm2") * self(p + "ls2")
        return x

    def chunk_attention(self, x, p, m):
        q, k, v = (self.mul(x, p + n) + self(p + n + ".b") for n in "qkv")
        q = _turn(self.norm(q, p + "q.norm").unflatten(-1, (m["heads"], -1)), m["rot"])
        k = _turn(self.norm(k, p + "k.norm").unflatten(-1, (m["kv_heads"], -1)), m["rot"])
        return self.mul(_attend(q, k, v.unflatten(-1, (m["kv_heads"], -1)), m["scale"], _chunk(m["mask"]["size"])), p + "o")

    def head_delta(self, x, p, m):
        q, k, v = self.filtered(x, p, m)
        keep = torch.exp(-torch.exp(self(p + "A_log")) * torch.nn.functional.softplus(self.mul(x, p + "a") + self(p + "dt_bias")))
        o = _memory(q, k, v, keep[..., None], beta=torch.sigmoid(self.mul(x, p + "b")))
        return self.mul(self.norm(o, p + "norm").flatten(2) * _silu(self.mul(x, p + "g")), p + "o")

    # -- the final norm and the logits
    def head(self, x):
        name = self.raw.get("architecture")
        if name is None:
            tied = self.raw["tie_word_embeddings"]
            return self.mul(self.norm(x, "model.norm.weight"), "model.embed_tokens.weight" if tied else "lm_head.weight")
        if name == "Luzitar":
            cap = self.raw["logit_softcap"]
            return cap * torch.tanh(self.mul(self.dyt(x, "final.norm"), "head") / cap)
        if name == "Rolevik":
            return self.mul(self.layer_norm(x, "final.norm"), "embed") * self.raw["logit_scale"]
        if name in ("Pilonex", "Bubalix"):
            return self.mul(_rms(x, self.eps) * (1.0 + self("final.norm")), "head")
        return self.mul(self.norm(x, "final.norm"), "embed") * self.raw.get("logit_scale", 1.0)
