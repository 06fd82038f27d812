"""What is timed: the work that users have this engine do, through its public entry points.

Three kinds of case, each a dict of plain values:

* ``step``: ONE batch through ``Engine.step``, the function that the scheduler, ``Model.generate`` and trace replay all
  go through: ``decode`` requests that bring one token each, with contexts of up to ``context`` tokens, beside
  ``prompts`` requests that bring a portion of up to ``tokens`` tokens behind ``past`` tokens in the cache. The logits
  of every request's last token come back; then the requests forget the step, so that a pass can be repeated.
* ``generation``: ``requests`` requests from nothing: their prompts of up to ``tokens`` tokens in one step, then
  ``steps`` decode steps with given tokens (as trace replay feeds them), then the requests are closed. The logits of
  every step come back. The only form that fits models whose layers keep a state per request.
* ``sample``: one token for each of ``rows`` rows of logits, through ``Sampler.sample``, greedy and sampled rows mixed.

``spread`` makes a batch ragged: request i of n has ``1 - spread * i / n`` of the largest length. Contexts and prompts
are random ids and the weights are random: the engine's work does not depend on their values. The model sizes are the
Qwen2.5 shapes of the benchmark (four layers of the largest one) and its sizes of the Vagulorn and Nezalorn designs.
"""
import json
import math
import os
import shutil
import tempfile
import zlib

import numpy as np
import torch

from nanoinfer_b200 import load_model
from nanoinfer_b200.config.model_config import write_config_json
from nanoinfer_b200.engine import StepEntry
from nanoinfer_b200.registry import config_from_json_dict, plan_for
from nanoinfer_b200.sampling import SampleRow, SamplingParams
from nanoinfer_b200.weights.safetensors_io import save_safetensors

F64 = torch.float64

_QWEN = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": 24, "hidden_size": 896,
         "num_attention_heads": 14, "num_key_value_heads": 2, "head_dim": 64, "intermediate_size": 4864, "vocab_size": 151936,
         "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": True, "max_position_embeddings": 32768,
         "use_sliding_window": False, "hidden_act": "silu", "torch_dtype": "bfloat16"}


def _vagulorn(w, h, d, ff, rot):
    half = {"heads": h, "kv_heads": 2, "dim": d, "vdim": d, "scale": d ** -0.5}
    pair = {"left": dict(half, mask={"size": 1024, "keep_first": 4}, rot={"dims": rot, "base": 500000.0}),
            "right": {"heads": 4, "dim": d, "vdim": d, "decay": [1.0 - 2.0 ** -(3 + 2 * i) for i in range(4)]},
            "left_scale": 1.0, "right_scale": 0.75}
    chunked = dict(half, mask={"size": 1024}, rot={"dims": rot, "base": 50000.0})
    ssm = {"heads": 32, "vdim": 2 * w // 32, "state": 128, "groups": 2, "norm_groups": 2, "conv": 4}
    mlp = {"kind": "dense", "ff": ff}
    kinds = [{"type": "parallel", "mixer": pair, "mlp": mlp}, {"type": "mamba2", "mixer": ssm, "mlp": mlp},
             {"type": "attention", "mixer": chunked, "mlp": mlp}]
    return {"architecture": "Vagulorn", "vocab": 32000, "width": w, "norm": {"eps": 1e-5}, "embedding": {"scale": 8.0},
            "layers": [kinds[(0, 1, 2, 1)[i % 4]] for i in range(8)]}


def _nezalorn(w, h, d, ff, rot, q_rank, blocks):
    mlp = {"kind": "dense", "ff": ff}
    lat = {"heads": h, "dim": d, "rot_dim": rot, "vdim": d, "q_rank": q_rank, "kv_rank": 128, "mask": {"size": 1024},
           "scale": (d + rot) ** -0.5,
           "rot": {"dims": rot, "base": 10000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    delta = {"type": "general_delta", "mixer": {"heads": h, "dim": d, "decay_rank": 64}, "mlp": mlp}
    lru = {"type": "rglru", "mixer": {"width": w, "conv": 4, "blocks": blocks}, "mlp": mlp}
    layers = []
    for i in range(8):
        layers.append((delta, lru, lru)[i % 4] if i % 4 < 3
                      else {"type": "latent_attention", "mixer": dict(lat) if i == 3 else dict(lat, kv_from=3), "mlp": mlp})
    return {"architecture": "Nezalorn", "vocab": 32000, "width": w, "norm": {"eps": 1e-5}, "layers": layers}


# name -> (configuration, cache tokens, live requests): the cache holds what four programs' worth of requests need
_MODELS = {
    "qwen2.5-0.5b": (_QWEN, 1 << 20, 288),
    "qwen2.5-1.5b": (dict(_QWEN, num_hidden_layers=28, hidden_size=1536, num_attention_heads=12, head_dim=128,
                          intermediate_size=8960), 1 << 19, 160),
    "qwen2.5-7b-4layers": (dict(_QWEN, num_hidden_layers=4, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4,
                                head_dim=128, intermediate_size=18944, vocab_size=152064, tie_word_embeddings=False),
                           1 << 19, 160),
    "vagulorn-1k": (_vagulorn(1024, 16, 64, 2816, 32), 1 << 16, 48),
    "vagulorn-2k": (_vagulorn(2048, 16, 128, 5632, 64), 1 << 16, 48),
    "nezalorn-1k": (_nezalorn(1024, 16, 64, 4224, 32, 384, 8), 1 << 16, 48),
    "nezalorn-2k": (_nezalorn(2048, 16, 128, 8448, 64, 768, 16), 1 << 16, 48),
}
_STD = {"matrix": 0.02, "embedding": 0.02, "bias": 0.02, "unit": 1.0}


def listed():
    q05, q15, q7 = "qwen2.5-0.5b", "qwen2.5-1.5b", "qwen2.5-7b-4layers"
    return [
        # one user's chat, a token at a time: nothing but latency
        _step("decode_1", q05, decode=1, context=777),
        # the benchmark's headline: eight users at a context of 4,096
        _step("decode_8_ctx4096", q05, decode=8, context=4090),
        # a loaded server: sixty-four users at very different places in their conversations
        _step("decode_64_ragged", q05, decode=64, context=4000, spread=0.95),
        # the headline at the family's next size (heads of 128)
        _step("decode_8_ctx4096_1.5b", q15, decode=8, context=4090),
        # a long question or a short document
        _step("prompt_2048", q05, prompts=1, tokens=2048),
        # a server's ordinary step: users that decode beside new prompts of odd lengths
        _step("mixed_24_and_3", q05, decode=24, context=1500, prompts=3, tokens=601, spread=0.7),
        # the last portion of a long document
        _step("prompt_2048_after_14k", q15, prompts=1, tokens=2048, past=14336),
        # two long prompts at the widths of the largest shape
        _step("prompts_2x4096_7b", q7, prompts=2, tokens=4096),
        # the 32-bit mode at the reference's own workload: a prompt of 128 tokens, then decoding
        {"name": "generate_f32", "kind": "generation", "model": q05, "dtype": "float32", "requests": 1, "tokens": 128, "steps": 16,
         "spread": 0.0},
        # the last step of every decode: draws for eight users
        {"name": "sample_8", "kind": "sample", "rows": 8, "vocab": 151936},
        # other designs, prompts and decoding: state-space mixers and lightning attention, delta rule and gated recurrences
        {"name": "generate_vagulorn", "kind": "generation", "model": "vagulorn-2k", "dtype": "bfloat16", "requests": 3, "tokens": 1100,
         "steps": 12, "spread": 0.5},
        {"name": "generate_nezalorn", "kind": "generation", "model": "nezalorn-1k", "dtype": "bfloat16", "requests": 3, "tokens": 1100,
         "steps": 12, "spread": 0.5},
    ]


def _step(name, model, dtype="bfloat16", decode=0, context=0, prompts=0, tokens=0, past=0, spread=0.0):
    return {"name": name, "kind": "step", "model": model, "dtype": dtype, "decode": decode, "context": context, "prompts": prompts,
            "tokens": tokens, "past": past, "spread": spread}


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    spread = round(rng.choice([0.0, rng.uniform(0.0, 0.95)]), 3)
    what = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "float32", "design", "sample"])
    model = rng.choice(["qwen2.5-0.5b", "qwen2.5-0.5b", "qwen2.5-1.5b", "qwen2.5-7b-4layers"])
    if what == "decode":
        c = _step("", model, decode=log(1, 64 if model == "qwen2.5-0.5b" else 24), context=log(17, 4090), spread=spread)
    elif what == "prompt":
        n = rng.choice([1, 1, 2, 3])
        c = _step("", model, prompts=n, tokens=log(9, 4096 // n), past=rng.choice([0, 0, log(16, 8192)]), spread=spread)
    elif what == "mixed":
        c = _step("", model, decode=log(1, 32), context=log(17, 2048), prompts=rng.choice([1, 2, 3]), tokens=log(9, 1000), spread=spread)
    elif what == "float32":
        c = {"kind": "generation", "model": "qwen2.5-0.5b", "dtype": "float32", "requests": rng.choice([1, 1, 2, 4]), "tokens": log(16, 256),
             "steps": log(4, 16), "spread": spread}
    elif what == "design":
        c = {"kind": "generation", "model": rng.choice(["vagulorn-1k", "vagulorn-2k", "nezalorn-1k", "nezalorn-2k"]), "dtype": "bfloat16",
             "requests": rng.choice([1, 2, 3, 4]), "tokens": log(32, 1400), "steps": log(4, 12), "spread": spread}
    else:
        c = {"kind": "sample", "rows": log(1, 64), "vocab": rng.choice([151936, 152064, 32000])}
    c.pop("name", None)
    return c


# ---- lengths, weights, models ----------------------------------------------------------------------------
def _lengths(n, largest, spread):
    return [max(1, int(largest * (1.0 - spread * i / n))) for i in range(n)]


def _requests(case):
    """[(tokens in the cache, tokens that the step brings)] of a ``step`` case."""
    out = [(c, 1) for c in _lengths(case["decode"], case["context"], case["spread"])] if case["decode"] else []
    return out + ([(case["past"], t) for t in _lengths(case["prompts"], case["tokens"], case["spread"])] if case["prompts"] else [])


_kept = {}


def _weights(name):
    """{tensor name: bfloat16 tensor on the GPU}: N(0, 0.02) matrices and biases, gains near 1, every tensor from a seed of its own."""
    if ("weights", name) not in _kept:
        out = {}
        for ts in plan_for(config_from_json_dict(_MODELS[name][0])).tensor_specs():
            g = torch.Generator(device="cuda").manual_seed(zlib.crc32(ts.name.encode()))
            x = torch.randn(ts.shape, generator=g, device="cuda")
            if ts.init == "gain":
                x = 1.0 + 0.1 * x
            elif ts.init == "mix":
                x = (1.0 + 0.3 * x) / max(1, x.numel())
            else:
                x = _STD[ts.init] * x
            out[ts.name] = x.to(torch.bfloat16)
        _kept["weights", name] = out
    return _kept["weights", name]


def _model(name, dtype):
    """A loaded model: a program loads one and keeps it for all its requests, and so do all cases on that model."""
    if (name, dtype) not in _kept:
        config, cache_tokens, live = _MODELS[name]
        folder = tempfile.mkdtemp(prefix="nanoinfer_b200_cases_")
        try:
            write_config_json(config_from_json_dict(config), folder)
            save_safetensors(os.path.join(folder, "model.safetensors"), _weights(name))
            _kept[name, dtype] = load_model(folder, dtype=dtype, page_size=16, num_pages=(cache_tokens if dtype == "bfloat16" else 1 << 16) // 16,
                                            max_batch=live, max_tokens_per_step=4096)
        finally:
            shutil.rmtree(folder, ignore_errors=True)
    return _kept[name, dtype]


class _Live:
    """A program's open requests and what its next step brings; they are closed with it."""
    count = steps = 0

    def __init__(self, model):
        self.model, self.engine, self.requests, self.entries = model, model.engine, [], []

    def open(self):
        _Live.count += 1
        self.requests.append(self.engine.open(f"case{_Live.count}"))
        return self.requests[-1]

    def __del__(self):
        for rc in self.requests:
            if not rc.closed:
                self.engine.close(rc)


def _tokens(case, seed):
    """The requests' token ids, host arrays as a tokenizer gives them; of a ``step`` case (in the cache, of the step)."""
    rng = np.random.default_rng(int(seed) * 2 + 1)
    vocab = _vocab(case["model"])
    if case["kind"] == "step":
        return [tuple(rng.integers(0, vocab, n).astype(np.int32) for n in pair) for pair in _requests(case)]
    return [(rng.integers(0, vocab, t).astype(np.int32), rng.integers(0, vocab, case["steps"]).tolist())
            for t in _lengths(case["requests"], case["tokens"], case["spread"])]


def _vocab(name):
    c = _MODELS[name][0]
    return c.get("vocab_size") or c["vocab"]


def _logit_rows(case, seed):
    """Logits as a trained model gives them: a few tokens far above a broad rest."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x = 2.0 * torch.randn(case["rows"], case["vocab"], generator=g, device="cuda")
    return x + 6.0 * (torch.rand(x.shape, generator=g, device="cuda") < 2e-4)


def _sample_rows(case, seed):
    kinds = [dict(temperature=0.7, top_p=0.9), dict(temperature=0.8, top_k=40), dict(temperature=1.0), dict(temperature=0.0),
             dict(temperature=0.9, top_k=50, top_p=0.95), dict(temperature=0.6, top_p=0.95)]
    return [SampleRow(SamplingParams(**kinds[i % len(kinds)]), None, 5 + i, seed=int(seed) + i) for i in range(case["rows"])]


# ---- what is timed ---------------------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "sample":
        return {"case": case, "model": _model("qwen2.5-0.5b", "bfloat16"), "logits": _logit_rows(case, seed), "rows": _sample_rows(case, seed)}
    model = _model(case["model"], case["dtype"])
    tokens = _tokens(case, seed)
    if case["kind"] == "generation":
        return {"case": case, "model": model, "tokens": tokens}
    live = _Live(model)
    jobs = [[live.open(), past, 0] for past, _ in tokens]
    # contexts are fed as a server feeds them, in portions under a budget; the portions' lengths differ, as prompts' do (the
    # engine keeps a few shapes of step that recur; these are not to be among them)
    while any(at < len(past) for _, past, at in jobs):
        _Live.steps += 1
        room, batch = 2048 + _Live.steps % 997, []
        for job in jobs:
            n = min(room, len(job[1]) - job[2])
            if n > 0:
                batch.append(StepEntry(job[0], job[1][job[2]:job[2] + n], []))
                job[2] += n
                room -= n
        live.engine.step(batch)
    live.entries = [StepEntry(job[0], new if len(new) > 1 else [int(new[0])], [len(new) - 1]) for job, (_, new) in zip(jobs, tokens)]
    live.lengths = [rc.length for rc in live.requests]
    return {"case": case, "model": model, "live": live}


def run(state):
    case, model = state["case"], state["model"]
    if case["kind"] == "sample":
        return torch.tensor(model.sampler.sample(state["logits"], state["rows"]))
    if case["kind"] == "step":
        live = state["live"]
        logits = live.engine.step(live.entries)
        for rc, n in zip(live.requests, live.lengths):
            live.engine.truncate(rc, n)
        return logits
    engine, live, out = model.engine, _Live(model), []
    requests = [live.open() for _ in state["tokens"]]
    out.append(engine.step([StepEntry(rc, prompt, [len(prompt) - 1]) for rc, (prompt, _) in zip(requests, state["tokens"])]))
    for s in range(case["steps"]):
        out.append(engine.step([StepEntry(rc, [given[s]], [0]) for rc, (_, given) in zip(requests, state["tokens"])]))
    for rc in requests:
        engine.close(rc)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------
def _attention_sizes(name):
    """(layers' list of (query heads, key heads, head size, window or 0)) of a model's softmax layers."""
    c = _MODELS[name][0]
    if name.startswith("qwen"):
        return [(c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], 0)] * c["num_hidden_layers"]
    out = []
    for layer in c["layers"]:
        m = layer["mixer"]
        m = m.get("left", m)
        if layer["type"] == "latent_attention":
            out.append((m["heads"], 1, m["dim"], m["mask"]["size"]))
        elif "kv_heads" in m:
            out.append((m["heads"], m["kv_heads"], m["dim"], m["mask"]["size"]))
    return out


def _step_work(case, pairs):
    c, size = _MODELS[case["model"]][0], 2 if case["dtype"] == "bfloat16" else 4
    tied = c.get("tie_word_embeddings", True)
    layer = head = 0
    for ts in plan_for(config_from_json_dict(c)).tensor_specs():
        n = math.prod(ts.shape)
        if ts.init == "embedding" or ts.name in ("embed", "model.embed_tokens.weight"):
            head += n if tied else 0
        elif ts.name == "lm_head.weight":
            head += n
        else:
            layer += n
    tokens, rows = sum(t for _, t in pairs), len(pairs)
    bytes_ = size * (layer + head) + 4 * rows * _vocab(case["model"])
    flops = 2.0 * layer * tokens + 2.0 * head * rows
    for q, kv, d, window in _attention_sizes(case["model"]):
        for past, t in pairs:
            seen = sum(min(past + i + 1, window or 1 << 30) for i in range(t)) if window else t * past + t * (t + 1) / 2.0
            flops += 4.0 * q * d * seen
            bytes_ += 2 * size * kv * d * (min(past, window or past) + t)
    return bytes_, flops


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4 * case["rows"] * (case["vocab"] + 1), "flops": 0}
    if case["kind"] == "step":
        b, f = _step_work(case, _requests(case))
        return {"bytes": b, "flops": f}
    lengths = _lengths(case["requests"], case["tokens"], case["spread"])
    steps = [[(0, t) for t in lengths]] + [[(t + s, 1) for t in lengths] for s in range(case["steps"])]
    done = [_step_work(case, p) for p in steps]
    return {"bytes": sum(b for b, _ in done), "flops": sum(f for _, f in done)}


def tolerance(case):
    """About four times what was seen against 64 bits in 32-bit mode (3.5e-6), and four times what two runs of one bfloat16
    step differ by (their sums go into the residual stream in any order: 0.002 to 0.01, at most 0.05 of a value's scale); a
    step's own distance from 64 bits is 0.004 to 0.017."""
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5, "max": 3e-4}
    return {"rel": 0.03, "max": 0.2}


# ---- the same in 64 bits, without the engine -------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "sample":
        return None
    c, w = _MODELS[case["model"]][0], _weights(case["model"])
    if case["kind"] == "step":
        seqs = [(np.concatenate([past, new]), [len(past) + len(new) - 1]) for past, new in _tokens(case, seed)]
    else:
        seqs = [(np.concatenate([p, np.asarray(g, np.int32)]), [len(p) - 1 + s for s in range(case["steps"] + 1)]) for p, g in _tokens(case, seed)]
    b, f = _step_work(case, [(0, len(ids)) for ids, _ in seqs])
    if f > 2e14:        # over about 20 seconds of 64-bit products
        return None
    forward = _exact_qwen if case["model"].startswith("qwen") else _exact_vagulorn if case["model"].startswith("vagulorn") else _exact_nezalorn
    with torch.no_grad():
        rows = [forward(c, w, torch.as_tensor(ids, dtype=torch.long, device="cuda"), places) for ids, places in seqs]
    if case["kind"] == "step":
        return torch.cat(rows)
    return [torch.stack([r[s] for r in rows]) for s in range(case["steps"] + 1)]


def _dot(h, w):
    return h @ w.to(F64).t()


def _rms(x, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    return _rms(x, eps) * w.to(F64) + b.to(F64)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _turn(x, freq, interleaved=False, mag=1.0):
    """x [T, heads, d]: the first 2 * len(freq) channels of every head turned by position."""
    n = freq.numel()
    a = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None, None] * freq
    c, s = a.cos() * mag, a.sin() * mag
    u, v = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if interleaved else (x[..., :n], x[..., n:2 * n])
    lo, hi = u * c - v * s, v * c + u * s
    turned = torch.stack([lo, hi], -1).flatten(-2) if interleaved else torch.cat([lo, hi], -1)
    return torch.cat([turned, x[..., 2 * n:]], -1)


def _freq(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device="cuda") / dims)


def _attend(q, k, v, scale, sees, block=512):
    """q [T, H, d], k and v [T, G, .]; ``sees(i, j)`` says which earlier positions j a position i reads."""
    t, heads, groups = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(t, heads, v.shape[2], dtype=F64, device=q.device)
    for a in range(0, t, block):
        e = min(t, a + block)
        i, j = torch.arange(a, e, device=q.device)[:, None], torch.arange(e, device=q.device)[None, :]
        hidden = ~((j <= i) & sees(i, j))
        for g in range(groups):
            hs = slice(g * heads // groups, (g + 1) * heads // groups)
            s = torch.einsum("thd,sd->hts", q[a:e, hs], k[:e, g]) * scale
            p = torch.softmax(s.masked_fill_(hidden, -math.inf), -1)
            out[a:e, hs] = torch.einsum("hts,sd->thd", p, v[:e, g])
    return out


def _exact_qwen(c, w, ids, places):
    eps, hd, nq, nkv = c["rms_norm_eps"], c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"]
    x = w["model.embed_tokens.weight"][ids].to(F64)
    t, freq = x.shape[0], _freq(hd, c["rope_theta"])
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w[p + "input_layernorm.weight"].to(F64)
        q, k, v = (_dot(h, w[f"{p}self_attn.{n}_proj.weight"]) + w[f"{p}self_attn.{n}_proj.bias"].to(F64) for n in "qkv")
        q, k = _turn(q.view(t, nq, hd), freq), _turn(k.view(t, nkv, hd), freq)
        o = _attend(q, k, v.view(t, nkv, hd), hd ** -0.5, lambda i, j: j <= i)
        x = x + _dot(o.reshape(t, -1), w[p + "self_attn.o_proj.weight"])
        h = _rms(x, eps) * w[p + "post_attention_layernorm.weight"].to(F64)
        x = x + _dot(_silu(_dot(h, w[p + "mlp.gate_proj.weight"])) * _dot(h, w[p + "mlp.up_proj.weight"]), w[p + "mlp.down_proj.weight"])
    h = _rms(x[places], eps) * w["model.norm.weight"].to(F64)
    return _dot(h, w["model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight"])


def _conv(u, w, bias):
    """u [T, C], w [C, taps]: a causal convolution per channel, the last tap on the token itself."""
    taps, t = w.shape[1], u.shape[0]
    padded = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    return bias.to(F64) + sum(padded[j:j + t] * w[:, j].to(F64) for j in range(taps))


def _matrix_state(q, k, v, decay):
    """S_t = decay_t S_(t-1) + k_t v_t^T and o_t = S_t^T q_t per head."""
    s = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=F64, device=k.device)
    out = torch.empty_like(v)
    for t in range(k.shape[0]):
        s = decay[t][:, None, None] * s + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.matmul(q[t][:, None, :], s)[:, 0]
    return out


def _exact_vagulorn(c, w, ids, places):
    eps = c["norm"]["eps"]
    x = w["embed"][ids].to(F64) * c["embedding"]["scale"]
    t = x.shape[0]

    def softmax(h, p, m, interleaved, sees):
        k = _dot(h, w[p + ".k"]).view(t, m["kv_heads"], m["dim"])
        v = k if interleaved else _dot(h, w[p + ".v"]).view(t, m["kv_heads"], m["vdim"])
        q = _rms(_dot(h, w[p + ".q"]).view(t, m["heads"], m["dim"]), eps) * w[p + ".q.norm"].to(F64)
        freq = _freq(m["rot"]["dims"], m["rot"]["base"])
        q, k = _turn(q, freq, interleaved), _turn(_rms(k, eps) * w[p + ".k.norm"].to(F64), freq, interleaved)
        o = _attend(q, k, v, m["scale"], sees)
        if interleaved:     # the windowed half: values are the keys, a gate per head
            o = o * torch.sigmoid(_dot(h, w[p + ".g"]))[:, :, None]
        return _dot(o.reshape(t, -1), w[p + ".o"])

    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix", layer["mixer"]
        h = _layer_norm(x, w[f"l{i}.norm1"], w[f"l{i}.norm1.b"], eps)
        if layer["type"] == "attention":
            size = m["mask"]["size"]
            y = softmax(h, p, m, False, lambda i, j: i // size == j // size)
        elif layer["type"] == "parallel":
            a, b = m["left"], m["right"]
            y = m["left_scale"] * softmax(h, p + ".left", a, True, lambda i, j: (i - j < a["mask"]["size"]) | (j < a["mask"]["keep_first"]))
            q, k, v = (_silu(_dot(h, w[f"{p}.right.{n}"])).view(t, b["heads"], -1) for n in "qkv")
            o = _matrix_state(q, k, v, torch.tensor(b["decay"], dtype=F64, device="cuda").expand(t, -1)).reshape(t, -1)
            o = _rms(o, eps) * w[p + ".right.norm"].to(F64) * torch.sigmoid(_dot(h, w[p + ".right.g"]))
            y = y + m["right_scale"] * _dot(o, w[p + ".right.o"])
        else:
            heads, n, groups = m["heads"], m["state"], m["groups"]
            inner = heads * m["vdim"]
            z, u, dt = torch.split(_dot(h, w[p + ".in"]), [inner, inner + 2 * groups * n, heads], 1)
            u = _silu(_conv(u, w[p + ".conv"], w[p + ".conv.b"]))
            u, b, g = torch.split(u, [inner, groups * n, groups * n], 1)
            u = u.reshape(t, heads, -1)
            b, g = (a.reshape(t, groups, n).repeat_interleave(heads // groups, 1) for a in (b, g))
            dt = torch.nn.functional.softplus(dt + w[p + ".dt_bias"].to(F64), threshold=1e9)
            y = _matrix_state(g, b, u * dt[:, :, None], torch.exp(-torch.exp(w[p + ".A_log"].to(F64)) * dt))
            y = (y + w[p + ".D"].to(F64)[:, None] * u).reshape(t, inner) * _silu(z)
            y = _rms(y.view(t, m["norm_groups"], -1), eps).reshape(t, inner) * w[p + ".norm"].to(F64)
            y = _dot(y, w[p + ".o"])
        f = f"l{i}.mlp."
        x = x + y + _dot(_gelu(_dot(h, w[f + "gate"])) * _dot(h, w[f + "up"]), w[f + "down"])
    return _dot(_layer_norm(x[places], w["final.norm"], w["final.norm.b"], eps), w["embed"])


def _yarn(rot):
    """(frequencies, factor on cos and sin) of a rotation whose long wavelengths are stretched."""
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
    freq = _freq(dims, base)

    def at(turns):
        return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return freq / sc["factor"] * ramp + freq * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _exact_nezalorn(c, w, ids, places):
    eps = c["norm"]["eps"]
    x = w["embed"][ids].to(F64)
    t, results, rows = x.shape[0], [x], {}
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        g = {n: v.to(F64) for n, v in w.items() if n.startswith(f"l{i}.")}
        h = _rms(x, eps) * g[f"l{i}.norm1"]
        if layer["type"] == "latent_attention":
            heads, d = m["heads"], m["dim"]
            freq, mag = _yarn(m["rot"])
            if "kv_from" not in m:
                z = h @ g[p + "dkv"].t()
                rows[i] = (_rms(z[:, :m["kv_rank"]], eps) * g[p + "dkv.norm"], _turn(z[:, None, m["kv_rank"]:], freq, True, mag))
            latent, kr = rows[m.get("kv_from", i)]
            q = ((_rms(h @ g[p + "dq"].t(), eps) * g[p + "dq.norm"]) @ g[p + "uq"].t()).view(t, heads, -1)
            q = torch.cat([q[..., :d], _turn(q[..., d:], freq, True, mag)], -1)
            k = torch.cat([(latent @ g[p + "uk"].t()).view(t, heads, d), kr.expand(-1, heads, -1)], -1)
            o = _attend(q, k, (latent @ g[p + "uv"].t()).view(t, heads, -1), m["scale"], lambda i, j: i - j < m["mask"]["size"])
            y = o.reshape(t, -1) @ g[p + "o"].t()
        elif layer["type"] == "general_delta":
            heads, d = m["heads"], m["dim"]
            r, k, v = ((h @ g[p + n].t()).view(t, heads, d) for n in "rkv")
            decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ g[p + "w1"].t()) @ g[p + "w2"].t() + g[p + "w0"])).view(t, heads, d)
            unit = k / torch.sqrt(k.pow(2).sum(-1, keepdim=True) + 1e-6)
            taken = torch.sigmoid(h @ g[p + "a"].t() + g[p + "a.b"]).view(t, heads, d) * unit
            s, o = torch.zeros(heads, d, d, dtype=F64, device="cuda"), torch.empty(t, heads, d, dtype=F64, device="cuda")
            for j in range(t):
                seen = torch.matmul(unit[j][:, None, :], s)
                s = decay[j][:, :, None] * s - taken[j][:, :, None] * seen + k[j][:, :, None] * v[j][:, None, :]
                o[j] = torch.matmul(r[j][:, None, :], s)[:, 0]
            y = (_rms(o, eps).reshape(t, -1) * g[p + "norm"] * torch.sigmoid(h @ g[p + "g"].t())) @ g[p + "o"].t()
        else:
            width, nb = m["width"], m["blocks"]
            u = _conv(h @ g[p + "x"].t() + g[p + "x.b"], g[p + "conv"], g[p + "conv.b"])
            ub = u.view(t, nb, -1)
            gr, gi = (torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, g[p + n]) + g[p + n + ".b"]).reshape(t, width) for n in ("ra", "ri"))
            a = torch.exp(-8.0 * gr * torch.nn.functional.softplus(g[p + "lam"], threshold=1e9))
            b = torch.sqrt(1.0 - a ** 2) * gi * u
            s, o = torch.zeros(width, dtype=F64, device="cuda"), torch.empty(t, width, dtype=F64, device="cuda")
            for j in range(t):
                s = a[j] * s + b[j]
                o[j] = s
            y = (o * _gelu(h @ g[p + "y"].t() + g[p + "y.b"])) @ g[p + "o"].t()
        f, out = f"l{i}.mlp.", x + y
        z = (_rms(x, eps) * g[f"l{i}.norm2"]) @ g[f + "up"].t() + g[f + "up.b"]
        act = g[f + "act"]
        z = act[0] * _rms(z, eps) + act[1] * _rms(z ** 2, eps) + act[2] * _rms(z ** 3, eps) + act[3]
        results.append(out + z @ g[f + "down"].t() + g[f + "down.b"])
        x = sum(g[f"l{i}.dwa"][j] * results[j] for j in range(i + 2))
    return _dot(_rms(x[places], eps) * w["final.norm"].to(F64), w["embed"])
