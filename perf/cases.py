"""What a user of this engine has it do, as cases that can be timed and compared.

A case is either a small workload of requests on one model ("serve") or one call of the sampler
("sample").  A "serve" case opens its requests, feeds their prompts in portions under a step budget
of 2,048 tokens (decoded tokens first, then prompts, oldest first: the order of the engine's
scheduler), then feeds given tokens one a step per request, as a replay does, and closes them; its
outputs are the logits of every place a scheduler would sample at.  Given tokens, and not the
sampled ones, keep two runs comparable: with random weights a sampled token is a matter of rounding.

The models are those of the repository's benchmark: Qwen3 layer sizes (0.6B whole; twelve layers of
the 4B sizes; 0.6B in the true 32-bit path) and two of the other designs, Kusolorn (windowed
attention, delta rule, matrix memory) and Malazen (biased attention beside gated linear attention,
latent attention, a loop over layers), at the two widths they are benchmarked at.
A program that serves a model keeps one engine for all its requests: ``prepare`` builds the engine
of a model once and hands it to every state of that model.
"""

from __future__ import annotations

import gc
import json
import math
import tempfile
from pathlib import Path

import numpy as np
import torch
import torch.nn.functional as F

from lockstep_b200 import Engine, StepEntry
from lockstep_b200.config import config_from_dict
from lockstep_b200.engine import expected_weights
from lockstep_b200.sampling import Sampler, SamplingParams

PAGE, BUDGET, WEIGHT_SEED = 16, 2048, 20
POOL_TOKENS = 41_000          # positions the page pool holds (over the live requests)
MAX_LIVE = 64


# ---------------------------------------------------------------------------
# models: the repository's benchmark configurations
# ---------------------------------------------------------------------------

def _qwen3(**sizes):
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": 28, "hidden_size": 1024,
            "num_attention_heads": 16, "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": 3072,
            "vocab_size": 151936, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": True,
            "max_position_embeddings": 40960, **sizes}


def _kusolorn(width, heads, linear_heads, ff, side):
    # (all feed-forwards dense: the benchmark's has routed ones in every other layer, where in bfloat16 a router's close call
    # makes two right implementations differ by a whole expert's output)
    att = {"heads": heads, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0, "v_mix": True,
           "mask": {"size": 1024, "keep_first": 4},
           "rot": {"dims": 64, "base": 1000000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 1024}}}
    delta = {"heads": heads, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4}
    lstm = {"heads": linear_heads, "dim": 128, "vdim": 128, "gate_cap": 15.0}
    kinds = [("mlstm", lstm), ("delta", delta), ("attention", att), ("mlstm", lstm), ("delta", delta), ("attention", att),
             ("mlstm", lstm), ("delta", delta)]
    return {"architecture": "Kusolorn", "vocab": 32768, "width": width, "norm": {"eps": 1e-5}, "max_positions": 4096,
            "token_side": {"dim": side},
            "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": ff}} for t, m in kinds]}


def _malazen(width, heads, linear_heads, ff):
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    par = {"left": {"heads": heads, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                    "q_temp": {"coef": 0.1, "every": 1024}},
           "right": {"heads": linear_heads, "dim": 128, "vdim": 128, "tau": 8.0, "decay_rank": 64},
           "left_scale": 1.0, "right_scale": 0.5}
    lat = {"heads": heads, "dim": 96, "rot_dim": 32, "vdim": 128, "kv_rank": 96, "scale": 128 ** -0.5,
           "mask": {"size": 1024}, "rot": {"dims": 32, "base": 1000000.0,
                                           "scaling": {"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0}}}
    kinds = [("parallel", par), ("latent_attention", lat), ("latent_attention", lat), ("parallel", par),
             ("parallel", par), ("latent_attention", lat)]
    return {"architecture": "Malazen", "vocab": 32768, "width": width, "norm": {"eps": 1e-5, "groups": 2},
            "max_positions": 4096, "loop": {"start": 1, "stop": 3, "times": 2},
            "layers": [{"type": t, "mixer": m, "mlp": mlp} for t, m in kinds]}


MODELS = {
    "qwen3-0.6b": _qwen3(),
    "qwen3-4b-12-layers": _qwen3(num_hidden_layers=12, hidden_size=2560, num_attention_heads=32, intermediate_size=9728),
    "kusolorn-1024": _kusolorn(1024, 8, 4, 4096, 128),
    "kusolorn-2048": _kusolorn(2048, 16, 8, 8192, 256),
    "malazen-1024": _malazen(1024, 8, 4, 3072),
    "malazen-2048": _malazen(2048, 16, 8, 6144),
}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _serve(name, model, dtype, requests, lo, hi, new):
    return {"name": name, "kind": "serve", "model": model, "dtype": dtype, "requests": requests, "prompt_from": lo,
            "prompt_to": hi, "new": new}


def listed():
    q, s, m = "qwen3-0.6b", "kusolorn-1024", "malazen-1024"
    return [
        # one person's short question: a small prompt, then a token a step; latency and launches are all there is
        _serve("one_short_chat", q, "bfloat16", 1, 23, 23, 24),
        # the same prompt length class that no step budget fills: an odd short prompt on its own (time to first token)
        _serve("short_prompt", q, "bfloat16", 1, 173, 173, 1),
        # the benchmark's prompt (time to first token of an ordinary document)
        _serve("prompt_2048", q, "bfloat16", 1, 2048, 2048, 1),
        # a long document, odd length, fed in portions of the step budget
        _serve("prompt_8k", q, "bfloat16", 1, 8111, 8111, 1),
        # the benchmark's headline: eight requests decoding at a context of about 4,096
        _serve("eight_long_contexts", q, "bfloat16", 8, 3930, 3990, 96),
        # a busy server: 64 requests with prompts of about 512, decoding together
        _serve("sixty_four_requests", q, "bfloat16", 64, 384, 640, 40),
        # a continuous batch: prompts of every length, portions of prompts beside decoded tokens
        _serve("continuous_batch", q, "bfloat16", 16, 64, 2048, 48),
        # the true 32-bit path, prompts and decoding
        _serve("float32_serving", q, "float32", 3, 300, 900, 12),
        # a larger model (wider products, four query heads a key head)
        _serve("larger_model", "qwen3-4b-12-layers", "bfloat16", 6, 150, 1500, 32),
        # the design of state rules beside windowed attention: a small continuous batch
        _serve("kusolorn_serving", s, "bfloat16", 4, 300, 1400, 32),
        # the design of latent attention and gated linear attention: a document, then an answer
        _serve("malazen_document", m, "bfloat16", 2, 1700, 2000, 24),
        # next tokens of a busy server's step, temperature and nucleus
        {"name": "sample_top_p", "kind": "sample", "rows": 64, "vocab": 151936, "temperature": 0.8, "top_p": 0.9},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_estimate(c) for c in listed())
    while True:
        case = _draw(rng)
        if _estimate(case) <= most:
            return case


def _draw(rng):
    kind = rng.choices(["qwen", "float32", "larger", "kusolorn", "malazen", "sample"], [6, 2, 1, 2, 2, 2])[0]
    if kind == "sample":
        top_p = rng.choice([1.0, round(rng.uniform(0.5, 0.99), 3)])
        return {"kind": "sample", "rows": _log(rng, 1, 64), "vocab": rng.choice([32768, 50257, 151936]),
                "temperature": round(rng.uniform(0.5, 1.2), 3), "top_p": top_p}
    model, dtype, requests, longest, new = {
        "qwen": ("qwen3-0.6b", "bfloat16", _log(rng, 1, 64), 8192, _log(rng, 1, 96)),
        "float32": ("qwen3-0.6b", "float32", _log(rng, 1, 8), 1024, _log(rng, 1, 24)),
        "larger": ("qwen3-4b-12-layers", "bfloat16", _log(rng, 1, 12), 2048, _log(rng, 1, 48)),
        "kusolorn": (rng.choice(["kusolorn-1024", "kusolorn-2048"]), "bfloat16", _log(rng, 1, 12), 2048, _log(rng, 1, 48)),
        "malazen": (rng.choice(["malazen-1024", "malazen-2048"]), "bfloat16", _log(rng, 1, 12), 2048, _log(rng, 1, 48)),
    }[kind]
    a, b = sorted((_log(rng, 5, longest), _log(rng, 5, longest)))
    while requests * (b + new) > 40_000:
        requests = max(1, requests // 2)
    return {"kind": "serve", "model": model, "dtype": dtype, "requests": requests, "prompt_from": a, "prompt_to": b, "new": new}


def _prompts(case):
    """Prompt lengths: spread evenly over the range, in an order that is neither rising nor falling."""
    n, lo, hi = case["requests"], case["prompt_from"], case["prompt_to"]
    even = [lo + (hi - lo) * i // max(1, n - 1) for i in range(n)]
    return sorted(even, key=lambda v: (v * 2654435761 % 4294967296, v))


def _plan(case):
    """The steps of a "serve" case: lists of (request, first position, tokens, whether its last place is wanted)."""
    prompts, new = _prompts(case), case["new"]
    n = len(prompts)
    held, given, steps = [0] * n, [0] * n, []
    while any(g < new for g in given):
        budget, step = BUDGET, []
        for i in range(n):
            if given[i] and given[i] < new:
                step.append((i, held[i], 1, True))
                budget -= 1
        for i in range(n):
            if held[i] < prompts[i] and budget > 0:
                take = min(budget, prompts[i] - held[i])
                step.append((i, held[i], take, held[i] + take == prompts[i]))
                budget -= take
        for i, _, take, want in step:
            held[i] += take
            given[i] += want
        steps.append(step)
    return steps


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _costs(model):
    """Weight elements of a step without its head, state elements of a request, flops of a token without attention and
    head, head elements, and for every layer that attends: elements of a cached position, flops per key that a token sees,
    window, first positions that stay visible."""
    cfg = MODELS[model]
    if "num_hidden_layers" in cfg:
        h, i, d, L = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"], cfg["num_hidden_layers"]
        nq, nkv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
        weights = L * ((nq + 2 * nkv) * d * h + h * nq * d + 3 * i * h)
        return {"weights": weights, "state": 0, "linear": 2 * weights, "head": cfg["vocab_size"] * h,
                "attend": [(2 * nkv * d, 4 * nq * d, 0, 0)] * L}
    w = cfg["width"]
    out = {"weights": 0, "state": 0, "linear": 0, "head": cfg["vocab"] * w, "attend": []}
    order = _order(cfg) if "loop" in cfg else [(i, False) for i in range(len(cfg["layers"]))]
    for i, _ in order:
        kind, m, ff = cfg["layers"][i]["type"], cfg["layers"][i]["mixer"], cfg["layers"][i]["mlp"]["ff"]
        rule = 0
        if kind == "attention":
            weights = w * (2 * m["heads"] + 2 * m["kv_heads"]) * 128
            out["attend"].append((2 * m["kv_heads"] * 128, 4 * m["heads"] * 128, m["mask"]["size"], m["mask"]["keep_first"]))
        elif kind == "delta":
            weights = w * ((3 * m["heads"] + 2 * m["kv_heads"]) * 128 + 2 * m["heads"])
            rule = m["heads"] * 128 * 128
            out["linear"] += 7 * rule
        elif kind == "mlstm":
            weights = w * (5 * m["heads"] * 128 + 2 * m["heads"])
            rule = m["heads"] * 128 * 128
            out["linear"] += 5 * rule
        elif kind == "parallel":
            a, b = m["left"], m["right"]
            weights = w * (2 * a["heads"] * 128 + 2 * a["kv_heads"] * 128 + 5 * b["heads"] * 128 + 64) + 64 * b["heads"] * 128
            rule = b["heads"] * 128 * 128
            out["linear"] += 5 * rule
            out["attend"].append((2 * a["kv_heads"] * 128, 4 * a["heads"] * 128, 0, 0))
        else:
            weights = w * (m["heads"] * 128 + 128 + m["heads"] * m["vdim"]) + 96 * m["heads"] * (96 + m["vdim"])
            out["attend"].append((128, 4 * m["heads"] * 128, m["mask"]["size"], 0))
        weights += (2 if "token_side" in cfg else 3) * ff * w + 2 * w * cfg.get("token_side", {}).get("dim", 0)
        out["weights"] += weights
        out["linear"] += 2 * weights
        out["state"] += rule
    return out


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4 * case["rows"] * case["vocab"], "flops": 0}
    c, size = _costs(case["model"]), 2 if case["dtype"] == "bfloat16" else 4
    vocab = MODELS[case["model"]].get("vocab_size") or MODELS[case["model"]]["vocab"]
    bytes_, flops = 0, 0
    for step in _plan(case):
        tokens, wanted = sum(t for _, _, t, _ in step), sum(w for _, _, _, w in step)
        bytes_ += size * (c["weights"] + (c["head"] if wanted else 0))
        bytes_ += 4 * wanted * vocab + 2 * 4 * c["state"] * len(step)
        flops += tokens * c["linear"] + 2 * wanted * c["head"]
        for row, per_key, window, kept in c["attend"]:
            for _, start, t, _ in step:
                first = max(0, start + 1 - window - kept) if window else 0
                bytes_ += size * row * (start - first + 2 * t)        # older keys read, the step's own written and read
                seen = sum(min(window + kept, p + 1) for p in range(start, start + t)) if window else t * (2 * start + t + 1) // 2
                flops += per_key * seen
    return {"bytes": bytes_, "flops": flops}


def _estimate(case):
    """Seconds, roughly, to keep drawn cases below the largest listed one."""
    w = work(case)
    if case["kind"] == "sample":
        return w["bytes"] / 1e11
    f32 = case["dtype"] == "float32"
    return w["bytes"] / 3e12 + w["flops"] / (2e13 if f32 else 5e14) + len(_plan(case)) * 1e-3


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.01}     # a draw that falls on the edge between two tokens
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.03, "max": 0.4}


# ---------------------------------------------------------------------------
# weights, engines, states
# ---------------------------------------------------------------------------

def _weights(model, dtype):
    """The model's tensors by name, from a fixed seed: matrices N(0, 0.02), gains 1 + N(0, 0.02), or what a part asks for."""
    kind = torch.bfloat16 if dtype == "bfloat16" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(WEIGHT_SEED)
    out = {}
    for name, spec in sorted(expected_weights(config_from_dict(MODELS[model]).model_spec()).items()):
        if spec.init is not None and spec.init[0] == "uniform":
            t = spec.init[1] + (spec.init[2] - spec.init[1]) * torch.rand(spec.shape, generator=gen, device="cuda")
        else:
            mean, std = spec.init[1:] if spec.init is not None else ((1.0, 0.02) if spec.role == "gain" else (0.0, 0.02))
            t = mean + std * torch.randn(spec.shape, generator=gen, device="cuda")
        out[name] = t.to(kind)
    return out


def _write_folder(folder, model, dtype):
    """A model folder: config.json and the tensors in the safetensors layout (a length, a JSON header, the bytes)."""
    (folder / "config.json").write_text(json.dumps(MODELS[model]))
    tensors, header, at = _weights(model, dtype), {}, 0
    for name, t in tensors.items():
        size = t.numel() * t.element_size()
        header[name] = {"dtype": "BF16" if dtype == "bfloat16" else "F32", "shape": list(t.shape), "data_offsets": [at, at + size]}
        at += size
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    with open(folder / "model.safetensors", "wb") as f:
        f.write(len(text).to_bytes(8, "little") + text)
        for t in tensors.values():
            t.reshape(-1).view(torch.uint8).cpu().numpy().tofile(f)


_engine: dict = {}      # the engine of the model in use


def _engine_of(model, dtype):
    if (model, dtype) not in _engine:
        _engine.clear()
        gc.collect()
        torch.cuda.empty_cache()
        with tempfile.TemporaryDirectory() as folder:
            _write_folder(Path(folder), model, dtype)
            _engine[model, dtype] = Engine(folder, dtype=dtype, device="cuda:0", num_pages=POOL_TOKENS // PAGE + 2 * MAX_LIVE,
                                           page_size=PAGE, max_running=MAX_LIVE, max_step_tokens=BUDGET,
                                           max_seq_len=min(8448, 40960 if "qwen" in model else 4096))
    return _engine[model, dtype]


def _tokens(case, seed):
    """The token ids of every request: its prompt and the tokens that are fed to it."""
    cfg = MODELS[case["model"]]
    rng = np.random.default_rng([seed, 7])
    return [rng.integers(0, cfg.get("vocab_size") or cfg["vocab"], n + case["new"] - 1).tolist() for n in _prompts(case)]


def prepare(case, seed):
    if case["kind"] == "sample":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        # a few likely tokens over a broad body, as a trained model's logits have
        logits = 2.0 * torch.randn(case["rows"], case["vocab"], generator=gen, device="cuda")
        logits[:, :50] += 4.0 * torch.rand(case["rows"], 50, generator=gen, device="cuda") + 5.0
        order = torch.rand(case["vocab"], generator=gen, device="cuda").argsort()
        logits = logits[:, order].contiguous()
        params = [SamplingParams(uid=f"request-{seed}-{i}", seed=i, temperature=case["temperature"], top_p=case["top_p"],
                                 position=100 + 17 * i) for i in range(case["rows"])]
        return {"sampler": Sampler(torch.device("cuda:0")), "logits": logits, "params": params}
    engine = _engine_of(case["model"], case["dtype"])
    steps = _plan(case)
    cfg = MODELS[case["model"]]
    rows = sum(want for step in steps for _, _, _, want in step)
    return {"engine": engine, "steps": steps, "tokens": _tokens(case, seed), "seed": seed,
            "logits": torch.empty(rows, cfg.get("vocab_size") or cfg["vocab"], device="cuda")}


def run(state):
    if "sampler" in state:
        return state["sampler"].sample_device(state["logits"], state["params"])
    runner, tokens, out = state["engine"].runner, state["tokens"], state["logits"]
    names = [f"{state['seed']}-{i}" for i in range(len(tokens))]
    for uid in names:
        runner.open(uid)
    row = 0
    for step in state["steps"]:
        entries = [StepEntry(uid=names[i], tokens=tokens[i][start:start + n], start=start, want=[n - 1] if want else [])
                   for i, start, n, want in step]
        logits = runner.step(entries, check=False, static_logits=True)
        out[row:row + len(logits)].copy_(logits)
        row += len(logits)
    for uid in names:
        runner.close(uid)
    return out


# ---------------------------------------------------------------------------
# the same in 64 bits, written out plainly
# ---------------------------------------------------------------------------

def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, angles, mag=1.0, pairs=False):
    """x [..., n, heads, d]: the first elements of every head turned by ``angles`` [n, half]."""
    half = angles.shape[1]
    c, s = (angles.cos() * mag)[:, None, :], (angles.sin() * mag)[:, None, :]
    if pairs:
        a, b = x[..., 0:2 * half:2], x[..., 1:2 * half:2]
        turned = torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    else:
        a, b = x[..., :half], x[..., half:2 * half]
        turned = torch.cat([a * c - b * s, b * c + a * s], -1)
    return torch.cat([turned, x[..., 2 * half:]], -1)


def _angles(n, dims, base):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    return torch.arange(n, dtype=torch.float64, device="cuda")[:, None] * f


def _attend(q, k, v, scale, window=0, bias=None, sink=None, kept=0, cap=None):
    """q [B, n, H, d], k, v [B, n, G, d] -> [B, n, H, dv]; query rows in blocks, one sequence at a time."""
    n, H = q.shape[1], q.shape[2]
    rep = H // k.shape[2]
    out = torch.empty(*q.shape[:3], v.shape[-1], dtype=q.dtype, device=q.device)
    keys = torch.arange(n, device=q.device)
    for b in range(q.shape[0]):
        kb, vb = k[b].repeat_interleave(rep, 1).permute(1, 2, 0), v[b].repeat_interleave(rep, 1).transpose(0, 1)
        for at in range(0, n, 1024):
            end = min(n, at + 1024)
            rows = torch.arange(at, end, device=q.device)
            s = q[b, at:end].transpose(0, 1) @ kb[..., :end] * scale
            s = s if cap is None else cap * torch.tanh(s / cap)
            gap = rows[:, None] - keys[None, :end]
            if bias is not None:
                s = s - bias[0][:, None, None] * torch.log1p(bias[1][:, None, None] * gap.clamp(min=0))
            seen = (gap >= 0) & ((gap < window) | (keys[None, :end] < kept) if window else True)
            s = s.masked_fill(~seen, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                top = torch.maximum(top, sink[:, None, None])
            e = torch.exp(s - top)
            total = e.sum(-1, keepdim=True)
            if sink is not None:
                total = total + torch.exp(sink[:, None, None] - top)
            out[b, at:end] = ((e / total) @ vb[:, :end]).transpose(0, 1)
    return out


def _qwen3_exact(cfg, w, x, ids):
    n, d, eps = x.shape[1], cfg["head_dim"], cfg["rms_norm_eps"]
    H, G = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    angles = _angles(n, d, cfg["rope_theta"])
    for i in range(cfg["num_hidden_layers"]):
        t = {k.split(".", 3)[3]: v for k, v in w.items() if k.startswith(f"model.layers.{i}.")}
        t = {k.replace(".weight", "").split(".")[-1]: v.double() for k, v in t.items()}
        y = _rms(x, eps) * t["input_layernorm"]
        q, k, v = (F.linear(y, t[s + "_proj"]).unflatten(-1, (-1, d)) for s in "qkv")
        q, k = _turn(_rms(q, eps) * t["q_norm"], angles), _turn(_rms(k, eps) * t["k_norm"], angles)
        x = x + F.linear(_attend(q, k, v, d ** -0.5).flatten(-2), t["o_proj"])
        y = _rms(x, eps) * t["post_attention_layernorm"]
        x = x + F.linear(F.silu(F.linear(y, t["gate_proj"])) * F.linear(y, t["up_proj"]), t["down_proj"])
    return _rms(x, eps) * w["model.norm.weight"].double()


def _before(x):
    """Every token's predecessor in its sequence; zeros before the first."""
    return F.pad(x, (0, 0, 1, 0))[:, :-1]


def _state_rule(q, k, v, decay, put=None, beta=None):
    """S <- decay S, then + k u^T with u = v (times ``put`` per head), or beta (v - S^T k); the result is S^T q.
    [B, n, H, d] each, decay [B, n, H, d] or [B, n, H, 1] -> [B, n, H, dv]."""
    S = torch.zeros(*q.shape[:1], q.shape[2], q.shape[3], v.shape[3], dtype=q.dtype, device=q.device)
    out = torch.empty(*q.shape[:3], v.shape[3], dtype=q.dtype, device=q.device)
    v = v if put is None else v * put[..., None]
    for t in range(q.shape[1]):
        S = decay[:, t, :, :, None] * S
        u = v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - (k[:, t, :, None, :] @ S)[..., 0, :])
        S = S + k[:, t, :, :, None] * u[..., None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :]
    return out


def _gelu(x):
    return F.gelu(x, approximate="tanh")


def _kusolorn_exact(cfg, w, x, ids):
    eps, n, first = cfg["norm"]["eps"], x.shape[1], None
    f = 1000000.0 ** (-2.0 * torch.arange(32, dtype=torch.float64, device=x.device) / 64)
    for i, layer in enumerate(cfg["layers"]):
        m, t = layer["mixer"], {k.split(".", 1)[1]: v.double() for k, v in w.items() if k.startswith(f"l{i}.")}
        y = _rms(x, eps) * t["norm1"]
        heads = lambda a, d=128: a.unflatten(-1, (-1, d))  # noqa: E731
        lin = lambda name: F.linear(y, t["mix." + name])  # noqa: E731
        if layer["type"] == "attention":
            sc = m["rot"]["scaling"]
            # wavelengths beyond original / low are stretched by the factor, those below original / high kept, a ramp between
            turns = sc["original"] * f / (2.0 * math.pi)
            ramp = ((turns - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
            angles = torch.arange(n, dtype=torch.float64, device=x.device)[:, None] * (f / sc["factor"] * (1 - ramp) + f * ramp)
            q, k = (_rms(_turn(heads(lin(s)), angles, 1.0, True), eps) for s in "qk")
            v = own = heads(lin("v"))
            if first is not None:
                v = (1.0 - t["mix.vmix"]) * own + t["mix.vmix"] * first
            first = own if first is None else first
            o = _attend(q, k, v, m["scale"], m["mask"]["size"], kept=m["mask"]["keep_first"], cap=m["softcap"]).flatten(-2)
        elif layer["type"] == "delta":
            def conv(a, taps):
                total = torch.zeros_like(a)
                for j in range(taps.shape[1] - 1, -1, -1):
                    total, a = total + a * taps[:, j], _before(a)
                return F.silu(total)
            q, k, v = (heads(conv(lin(s), t[f"mix.{s}.conv"])) for s in "qkv")
            unit = lambda a: a * torch.rsqrt((a * a).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
            rep = m["heads"] // m["kv_heads"]
            q, k = (unit(q) * 128 ** -0.5).repeat_interleave(rep, 2), unit(k).repeat_interleave(rep, 2)
            decay = torch.exp(-torch.exp(t["mix.A_log"]) * F.softplus(lin("a") + t["mix.dt_bias"], threshold=60.0))
            o = _rms(_state_rule(q, k, v, decay[..., None], beta=torch.sigmoid(lin("b"))), eps) * t["mix.norm"]
            o = o.flatten(-2) * F.silu(lin("g"))
        else:
            cap = m["gate_cap"]
            q, k, v = (heads(lin(s)) for s in "qkv")
            put = cap * torch.tanh((lin("i") + t["mix.i.b"]) / cap)
            keep = F.logsigmoid(cap * torch.tanh((lin("f") + t["mix.f.b"]) / cap))
            top = [torch.zeros_like(put[:, 0])]                  # the running maximum that the gates are measured from
            for j in range(n):
                top.append(torch.maximum(keep[:, j] + top[-1], put[:, j]))
            before, top = torch.stack(top[:-1], 1), torch.stack(top[1:], 1)
            # the memory and, as one more value of 1, the normaliser
            o = _state_rule(q * 128 ** -0.5, k, F.pad(v, (0, 1), value=1.0), torch.exp(keep + before - top)[..., None],
                            put=torch.exp(put - top))
            o = o[..., :-1] / (torch.maximum(o[..., -1:].abs(), torch.exp(-top)[..., None]) + 1e-6)
            o = _rms(o, eps).flatten(-2) * t["mix.norm"] * torch.sigmoid(lin("g"))
        x = x + F.linear(o, t["mix.o"])
        y = _rms(x, eps) * t["norm2"]
        x = x + F.linear(_gelu(F.linear(y, t["mlp.up"])), t["mlp.down"])
        dim = cfg["token_side"]["dim"]
        own = w["side.embed"][ids][..., i * dim:(i + 1) * dim].double()
        x = x + _rms(F.linear(_gelu(F.linear(x, t["side.gate"])) * own, t["side.proj"]), eps) * t["side.norm"]
    return _rms(x, eps) * w["final.norm"].double()


def _order(cfg):
    """The layers in the order they run, and whether the embedding is added before them."""
    a, b, times = (cfg["loop"][s] for s in ("start", "stop", "times"))
    again = [(i, turn > 0 and i == a) for turn in range(times) for i in range(a, b)]
    return [(i, False) for i in range(a)] + again + [(i, False) for i in range(b, len(cfg["layers"]))]


def _malazen_exact(cfg, w, x, ids):
    eps, n = cfg["norm"]["eps"], x.shape[1]
    norm = lambda a, gain: _rms(a.unflatten(-1, (cfg["norm"]["groups"], -1)), eps).flatten(-2) * gain  # noqa: E731
    heads = lambda a, d: a.unflatten(-1, (-1, d))  # noqa: E731
    x0 = x
    for i, add in _order(cfg):
        layer = cfg["layers"][i]
        m, t = layer["mixer"], {k.split(".", 1)[1]: v.double() for k, v in w.items() if k.startswith(f"l{i}.")}
        x = x + x0 if add else x
        y = norm(x, t["norm1"])
        lin = lambda name, a=y: F.linear(a, t["mix." + name])  # noqa: E731
        if layer["type"] == "parallel":
            a, b = m["left"], m["right"]
            q, k, v = (heads(lin(f"left.{s}") + t[f"mix.left.{s}.b"], 128) for s in "qkv")
            at = torch.arange(n, device=x.device)
            temp = 1.0 + a["q_temp"]["coef"] * torch.log(((at + 1) // a["q_temp"]["every"] + 1).double())
            o = _attend(q * temp[:, None, None], k, v, a["scale"], bias=(t["mix.left.r1"], t["mix.left.r2"])).flatten(-2)
            left = lin("left.o", o) + t["mix.left.o.b"]
            q, k, v = (heads(lin("right." + s), 128) for s in "qkv")
            decay = torch.exp(F.logsigmoid(heads(lin("right.a2", lin("right.a1")) + t["mix.right.a2.b"], 128)) / b["tau"])
            o = _rms(_state_rule(q * 128 ** -0.5, k, v, decay), eps) * t["mix.right.norm"]
            x = x + m["left_scale"] * left + m["right_scale"] * lin("right.o", o.flatten(-2) * F.silu(lin("right.g")))
        else:
            d, dr, rank, rot = m["dim"], m["rot_dim"], m["kv_rank"], m["rot"]
            sc = rot["scaling"]
            turn = lambda turns: dr * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))  # noqa: E731
            lo, hi = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), dr - 1)
            ramp = ((torch.arange(dr // 2, device=x.device).double() - lo) / max(hi - lo, 0.001)).clamp(0, 1)
            angles, mag = _angles(n, dr, rot["base"]) * (ramp / sc["factor"] + 1 - ramp), 0.1 * math.log(sc["factor"]) + 1
            q, down = heads(lin("q"), d + dr), lin("dkv")
            q = torch.cat([q[..., :d], _turn(q[..., d:], angles, mag, True)], -1)
            c = _rms(down[..., :rank], eps) * t["mix.dkv.norm"]
            turned = _turn(down[..., None, rank:], angles, mag, True).expand(*q.shape[:3], dr)
            k = torch.cat([heads(lin("uk", c), d), turned], -1)
            o = _attend(q, k, heads(lin("uv", c), m["vdim"]), m["scale"], m["mask"]["size"], sink=t["mix.sink"])
            x = x + lin("o", o.flatten(-2))
        y, limit = norm(x, t["norm2"]), layer["mlp"]["limit"]
        g = (F.linear(y, t["mlp.gate"]) + t["mlp.gate.b"]).clamp(max=limit)
        u = (F.linear(y, t["mlp.up"]) + t["mlp.up.b"]).clamp(-limit, limit)
        x = x + F.linear(g * torch.sigmoid(1.702 * g) * (u + 1.0), t["mlp.down"]) + t["mlp.down.b"]
    return norm(x, w["final.norm"].double())


def exact(case, seed):
    if case["kind"] == "sample":
        return None               # whole numbers: tokens
    cfg, w, tokens = MODELS[case["model"]], _weights(case["model"], case["dtype"]), _tokens(case, seed)
    forward = {"q": _qwen3_exact, "k": _kusolorn_exact, "m": _malazen_exact}[case["model"][0]]
    table = w["model.embed_tokens.weight" if "model.norm.weight" in w else "embed"]
    # sequences side by side, padded at their ends (a token sees none after it), as many as a few thousand tokens allow
    hidden, group = [None] * len(tokens), []
    order = sorted(range(len(tokens)), key=lambda i: len(tokens[i]))
    for j, i in enumerate(order):
        group.append(i)
        if j + 1 == len(order) or (len(group) + 1) * len(tokens[order[j + 1]]) > 8192:
            n = max(len(tokens[i]) for i in group)
            ids = torch.tensor([tokens[i] + [0] * (n - len(tokens[i])) for i in group], device="cuda")
            y = forward(cfg, w, table[ids].double(), ids)
            for k, i in enumerate(group):
                hidden[i] = y[k]
            group = []
    rows = [hidden[i][start + n - 1] for step in _plan(case) for i, start, n, want in step if want]
    return F.linear(torch.stack(rows), w.get("head", table).double())
