"""The work that programs have this engine do, as cases that can be timed and compared.

A case is one round of service by :meth:`kappai_b200.ModelRunner.step`, the one step function that everything in the
engine drives: some requests arrive together, their prompts are fed in steps of at most ``budget`` tokens (a request that
is through its prompt decodes beside the prompts that still run, as the scheduler orders a step: decoded tokens first),
every request decodes ``new`` tokens, and each ends when it has them.  Token ids are given, as when a text is scored or a
recorded trace is replayed, so that two implementations run the same inputs all the way; the logits of every step are
kept.  With ``score`` the logits at every place of the prompts are wanted.  With ``sample`` every step's tokens are
drawn on the device as well (temperature 0.8, top-k 40, top-p 0.9, min-p 0.1), one batched call a step.

Requests arrive one (``requests`` = 1) or several at a time; then their prompts differ in length, evenly from half to one
and a half times ``prompt``.  The models are the LFM2 shapes of 350M, 1.2B and 2.6B parameters and four layers of the
Tupalorn design (a state space mixer, retention, attention, attention through a window), random weights.
"""
import hashlib
import json
import math
import os
import struct
import tempfile
from functools import lru_cache

import numpy as np
import torch

from kappai_b200 import ModelRunner, SamplingParams, StepEntry
from kappai_b200.sampling.sampler import sample
from kappai_b200.weights import random_weights, save_safetensors

VOCAB = 65536
LFM2_1P2B = dict(
    architectures=["Lfm2ForCausalLM"], vocab_size=VOCAB, hidden_size=2048, num_hidden_layers=16, num_attention_heads=32,
    num_key_value_heads=8,
    layer_types=["conv", "conv", "full_attention", "conv", "conv", "full_attention", "conv", "conv", "full_attention", "conv",
                 "full_attention", "conv", "full_attention", "conv", "full_attention", "conv"],
    max_position_embeddings=128000, norm_eps=1e-5, conv_L_cache=3, conv_bias=False, block_ff_dim=8192,
    block_auto_adjust_ff_dim=True, block_ffn_dim_multiplier=1.0, block_multiple_of=256, rope_theta=1000000.0, tie_embedding=True)


def _tupalorn():
    width, heads, groups, dim, ff = 2048, 32, 8, 64, 5632
    ssm = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
    ret = {"heads": heads, "dim": dim, "vdim": dim, "decay": [1.0 - 2.0 ** (-3 - 6 * h / (heads - 1)) for h in range(heads)],
           "rot": {"dims": dim, "base": 10000.0}}
    att = {"heads": heads, "kv_heads": groups, "dim": dim, "vdim": dim, "scale": dim ** -0.5}
    mixers = [("mamba2", ssm), ("retention", ret), ("attention", dict(att, mask={"size": 8192})),
              ("attention", dict(att, kv_from=2, mask={"size": 1024}))]
    return {"architecture": "Tupalorn", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "logit_softcap": 50.0,
            "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}} for t, m in mixers]}


MODELS = {
    "lfm2-350m": (dict(LFM2_1P2B, hidden_size=1024, num_attention_heads=16, block_ff_dim=6656), 4),
    "lfm2-1.2b": (LFM2_1P2B, 2),
    "lfm2-2.6b": (dict(LFM2_1P2B, num_hidden_layers=30, block_ff_dim=10752,
                       layer_types=["full_attention" if i in (2, 6, 10, 14, 18, 21, 24, 27) else "conv" for i in range(30)]), 3),
    "tupalorn": (_tupalorn(), 2),
}
SAMPLING = SamplingParams(temperature=0.8, top_k=40, top_p=0.9, min_p=0.1, seed=4)


def _case(name, model, dtype, requests, prompt, new, budget=2048, score=False, sample=False):
    return {"name": name, "model": model, "dtype": dtype, "requests": requests, "prompt": prompt, "new": new,
            "budget": budget, "score": score, "sample": sample}


def listed():
    return [
        # a short question to a small model: latency of the smallest calls
        _case("chat_350m", "lfm2-350m", "bfloat16", 1, 9, 24),
        # one user at a time
        _case("single_1.2b", "lfm2-1.2b", "bfloat16", 1, 600, 64),
        # a few users at once
        _case("few_1.2b", "lfm2-1.2b", "bfloat16", 8, 700, 64),
        # a loaded server: prompts of many lengths beside decoding requests
        _case("serve_1.2b", "lfm2-1.2b", "bfloat16", 64, 150, 32),
        # a batch job on a small model
        _case("batch_350m", "lfm2-350m", "bfloat16", 200, 48, 16),
        # time to the first token: a short question, a page of text
        _case("first_token_101", "lfm2-1.2b", "bfloat16", 1, 101, 0),
        _case("first_token_2048", "lfm2-1.2b", "bfloat16", 1, 2048, 0),
        # a long document, fed in portions
        _case("document_2.6b", "lfm2-2.6b", "bfloat16", 1, 12001, 0),
        # texts are scored: the logits of every place
        _case("score_350m", "lfm2-350m", "bfloat16", 3, 333, 0, score=True),
        # the true 32-bit path: one request, and several with sampling
        _case("single_1.2b_f32", "lfm2-1.2b", "float32", 1, 513, 12),
        _case("few_350m_f32", "lfm2-350m", "float32", 8, 75, 24, sample=True),
        # recurrent mixers
        _case("few_tupalorn", "tupalorn", "bfloat16", 6, 501, 32),
    ]


# what draw() spreads over: (model, dtype, requests, prompt, new, score, sample), each size from ... to
RANGES = [
    ("lfm2-350m", "bfloat16", (1, 200), (5, 700), (8, 32), False, False),
    ("lfm2-1.2b", "bfloat16", (1, 64), (16, 700), (16, 64), False, False),
    ("lfm2-1.2b", "bfloat16", (1, 1), (48, 4096), (0, 0), False, False),
    ("lfm2-2.6b", "bfloat16", (1, 1), (1500, 12001), (0, 16), False, False),
    ("lfm2-350m", "bfloat16", (1, 8), (30, 600), (0, 0), True, False),
    ("lfm2-1.2b", "float32", (1, 4), (20, 513), (4, 12), False, False),
    ("lfm2-350m", "float32", (1, 8), (20, 300), (8, 24), False, True),
    ("tupalorn", "bfloat16", (1, 8), (60, 700), (8, 32), False, False),
]


def draw(rng):
    spread = lambda lo, hi: lo if lo == hi else min(hi, int(round(math.exp(rng.uniform(math.log(max(lo, 1)), math.log(hi))))))
    model, dtype, requests, prompt, new, score, sampled = rng.choice(RANGES)
    n = spread(*requests)
    # (many requests share the prompts' tokens: no case has more than 12,001 of them)
    c = _case("", model, dtype, n, spread(prompt[0], max(prompt[0], min(prompt[1], 12001 // n))), spread(*new),
              rng.choice((512, 1024, 2048)), score, sampled)
    del c["name"]
    return c


def prompt_lengths(case):
    n, p = case["requests"], case["prompt"]
    return [p] if n == 1 else [max(1, p // 2 + (p * i) // (n - 1)) for i in range(n)]


def plan(case):
    """The steps of the round: for each a list of (request, first token, tokens), decoded tokens first."""
    lengths, new, steps = prompt_lengths(case), case["new"], []
    at = [0] * len(lengths)
    while any(at[i] < n + new for i, n in enumerate(lengths)):
        step = [(i, at[i], 1) for i, n in enumerate(lengths) if n <= at[i] < n + new]
        left = case["budget"] - len(step)
        for i, n in enumerate(lengths):
            if at[i] < n and left > 0:
                m = min(n - at[i], left)
                step.append((i, at[i], m))
                left -= m
        for i, _, m in step:
            at[i] += m
        steps.append(step)
    return steps


def wanted(case, lengths, i, first, n):
    """Places of a request's portion whose logits are wanted: all, or those from the prompt's last token on."""
    return [j for j in range(n) if case["score"] or first + j >= lengths[i] - 1]


def tokens_of(case, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, VOCAB, n + case["new"]).tolist() for n in prompt_lengths(case)]


def model_folder(model):
    """A folder with the model's random weights, written once.  In the LFM2 shapes the embedding is 32 times and every
    sublayer's last matrix an eighth of what random weights have, so that the residual is the token's row and what the layers
    add to it in about equal parts, as in a trained model, and not the last layers' doing alone."""
    config, seed = MODELS[model]
    key = hashlib.sha256(json.dumps([config, seed], sort_keys=True).encode()).hexdigest()[:12]
    folder = os.path.join(tempfile.gettempdir(), f"kappai_b200_perf_{os.getuid()}_{key}")
    if not os.path.isdir(folder):
        part = tempfile.mkdtemp(prefix=os.path.basename(folder) + "_", dir=tempfile.gettempdir())
        tensors = random_weights(config, seed)
        if model != "tupalorn":
            for name, t in tensors.items():
                if name == "model.embed_tokens.weight":
                    t *= 32.0
                elif name.endswith(("out_proj.weight", "w2.weight")):
                    t *= 0.125
        save_safetensors(os.path.join(part, "model.safetensors"), tensors)
        with open(os.path.join(part, "config.json"), "w") as f:
            json.dump(config, f)
        try:
            os.rename(part, folder)
        except OSError:                     # another process was first
            return part
    return folder


@lru_cache(maxsize=None)
def runner_for(model, dtype):
    """A program loads its model once and keeps it; requests of all rounds share its cache."""
    return ModelRunner(model_folder(model), dtype=dtype, max_tokens=65536, max_requests=256, page_size=64, max_model_len=16384)


class Round:
    pass


def prepare(case, seed):
    s = Round()
    s.runner = runner_for(case["model"], case["dtype"])
    lengths, tokens = prompt_lengths(case), tokens_of(case, seed)
    base = [0]
    for n in lengths:
        base.append(base[-1] + (n if case["score"] else 1) + case["new"])
    s.steps = []
    for step in plan(case):
        entries, rows, sampled = [], [], []
        for i, first, n in step:
            want = wanted(case, lengths, i, first, n)
            entries.append(StepEntry(i, tokens[i][first:first + n], want))
            rows += [base[i] + first + j - (0 if case["score"] else lengths[i] - 1) for j in want]
            sampled += [first + j - lengths[i] + 1 for j in want]
        ended = [i for i, first, n in step if first + n == lengths[i] + case["new"]]
        s.steps.append((entries, torch.tensor(rows, dtype=torch.long, device="cuda"), rows, sampled, ended))
    s.logits = torch.empty((base[-1], VOCAB), dtype=torch.float32, device="cuda")
    s.tokens = torch.empty(base[-1], dtype=torch.int32, device="cuda") if case["sample"] else None
    return s


def run(s):
    for entries, at, rows, sampled, ended in s.steps:
        logits = s.runner.step(entries)
        if rows:
            s.logits.index_copy_(0, at, logits)
            if s.tokens is not None:
                s.tokens.index_copy_(0, at, sample(logits, [SAMPLING] * len(rows), [4 + r for r in rows], sampled))
        for i in ended:
            s.runner.end(i)
    return {"logits": s.logits} if s.tokens is None else {"logits": s.logits, "tokens": s.tokens}


# ------------------------------------------------------------------------------------------ what a round cannot do without

def _sizes(model):
    """(parameters of the matrices that every token meets, values of the cache a token, attention's score and value
    multiplications a token and key, values of fixed-size state a request)."""
    c = MODELS[model][0]
    if model == "tupalorn":
        d, ff, inner, n = c["width"], 5632, 4096, 128
        ssm, ret, own, borrowed = d * (3 * inner + 2 * n + 64), 5 * d * d, d * (2 * d + 2 * 512 + 32), d * (2 * d + 32)
        return ssm + ret + own + borrowed + 4 * 3 * d * ff, 2 * 512, 2 * 2 * 2 * d, 64 * 64 * n + 32 * 64 * 64 + 3 * (inner + 2 * n)
    d, H, G = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"]
    hd, ff, n_att = d // H, feed_forward_width(c), c["layer_types"].count("full_attention")
    n_conv = len(c["layer_types"]) - n_att
    return ((n_conv * 4 * d * d + n_att * (2 * d * d + 2 * d * G * hd) + (n_att + n_conv) * 3 * d * ff), n_att * 2 * G * hd,
            n_att * 2 * 2 * d, n_conv * 2 * d)


def work(case):
    matrices, cache, att, state = _sizes(case["model"])
    d = MODELS[case["model"]][0].get("hidden_size", 2048)
    size = 4 if case["dtype"] == "float32" else 2
    lengths, nbytes, flops = prompt_lengths(case), 0, 0
    for step in plan(case):
        n_out = sum(len(wanted(case, lengths, i, first, n)) for i, first, n in step)
        nbytes += size * (matrices + (VOCAB * d if n_out else 0)) + 4 * VOCAB * n_out
        flops += 2 * VOCAB * d * n_out
        for i, first, n in step:
            nbytes += size * cache * (first + n) + 4 * 2 * state
            flops += 2 * matrices * n + att * (n * first + n * (n + 1) // 2)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # Measured: two ways of cutting a bfloat16 round, which split the sums differently, are 0.0017 to 0.005 of the logits'
    # norm apart (largest single difference 0.01 to 0.024 of their root mean square), each 0.002 to 0.007 from 64 bits;
    # float32 is 0.7e-6 to 1.4e-6 from 64 bits.  A token sampled from float32 logits may meet a tie.
    if case["dtype"] == "float32":
        return {"rel": 6e-6, "max": 2e-4, "differ": 0.01}
    return {"rel": 0.02, "max": 0.1}


# ------------------------------------------------------------------------------------------ the same in 64 bits, plain torch

def feed_forward_width(c):
    ff, m = int(c["block_ffn_dim_multiplier"] * ((2 * c["block_ff_dim"]) // 3)), c["block_multiple_of"]
    return m * ((ff + m - 1) // m)


def read_weights(folder):
    with open(os.path.join(folder, "model.safetensors"), "rb") as f:
        (n,) = struct.unpack("<Q", f.read(8))
        header, data = json.loads(f.read(n)), np.frombuffer(f.read(), dtype=np.uint8)
    out = {}
    for name, e in header.items():
        if name != "__metadata__":
            raw = torch.from_numpy(data[e["data_offsets"][0]:e["data_offsets"][1]].copy())
            out[name] = raw.view({"BF16": torch.bfloat16, "F32": torch.float32}[e["dtype"]]).reshape(e["shape"]).cuda().double()
    return out


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def rotate(x, base):
    """x [T, heads, dim]: dimension i is paired with i + dim/2, the angle of position p is p base^(-2i/dim)."""
    half = x.shape[-1] // 2
    f = float(base) ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def attend(q, k, v, scale, window):
    T, H, _ = q.shape
    q, k, v = q.transpose(0, 1), k.repeat_interleave(H // k.shape[1], 1).transpose(0, 1), v.repeat_interleave(H // v.shape[1], 1).transpose(0, 1)
    out = []
    for lo in range(0, T, 512):
        hi = min(T, lo + 512)
        s = (q[:, lo:hi] @ k[:, :hi].transpose(1, 2)) * scale
        gap = torch.arange(lo, hi, device=q.device)[:, None] - torch.arange(hi, device=q.device)[None, :]
        out.append(torch.softmax(s.masked_fill((gap < 0) | (gap >= window), -math.inf), -1) @ v[:, :hi])
    return torch.cat(out, 1).transpose(0, 1)


def convolve(u, taps, bias=None):
    """y[t, c] = sum_j taps[c, j] u[t - (K - 1) + j, c]: zero before the sequence."""
    K = taps.shape[-1]
    up = torch.cat([u.new_zeros(K - 1, u.shape[1]), u])
    y = sum(up[j:j + u.shape[0]] * taps.reshape(-1, K)[:, j] for j in range(K))
    return y if bias is None else y + bias


def decayed_sums(q, k, v, log_a):
    """o_t = S_t^T q_t, S_t = a_t S_(t-1) + k_t v_t^T, in chunks; q, k [T, H, N], v [T, H, P], log_a [T, H]."""
    T, H, N = q.shape
    S, out = q.new_zeros(H, N, v.shape[2]), []
    for lo in range(0, T, 64):
        qc, kc, vc, c = (t[lo:lo + 64].transpose(0, 1) for t in (q, k, v, log_a.unsqueeze(-1)))
        c = torch.cumsum(c, 1)                                                       # [H, n, 1]
        w = torch.exp(torch.tril(c - c.transpose(1, 2))).tril()
        out.append((qc @ kc.transpose(1, 2) * w) @ vc + torch.exp(c) * (qc @ S))
        S = torch.exp(c[:, -1:]) * S + (kc * torch.exp(c[:, -1:] - c)).transpose(1, 2) @ vc
    return torch.cat(out, 1).transpose(0, 1)


def lfm2_hidden(w, c, tokens):
    d, H, G, eps = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["norm_eps"]
    hd, T, x = d // H, len(tokens), w["model.embed_tokens.weight"][tokens]
    for i, kind in enumerate(c["layer_types"]):
        m = {k[len(f"model.layers.{i}."):]: v for k, v in w.items() if k.startswith(f"model.layers.{i}.")}
        h = rms(x, eps) * m["operator_norm.weight"]
        if kind == "conv":
            b, g, u = (h @ m["conv.in_proj.weight"].T).split(d, 1)
            x = x + (g * convolve(b * u, m["conv.conv.weight"])) @ m["conv.out_proj.weight"].T
        else:
            q, k, v = ((h @ m[f"self_attn.{n}_proj.weight"].T).reshape(T, -1, hd) for n in "qkv")
            q = rotate(rms(q, eps) * m["self_attn.q_layernorm.weight"], c["rope_theta"])
            k = rotate(rms(k, eps) * m["self_attn.k_layernorm.weight"], c["rope_theta"])
            x = x + attend(q, k, v, hd ** -0.5, 1 << 40).reshape(T, d) @ m["self_attn.out_proj.weight"].T
        h = rms(x, eps) * m["ffn_norm.weight"]
        x = x + (torch.nn.functional.silu(h @ m["feed_forward.w1.weight"].T) * (h @ m["feed_forward.w3.weight"].T)) @ m["feed_forward.w2.weight"].T
    return rms(x, eps) * w["model.embedding_norm.weight"]


def tupalorn_hidden(w, c, tokens):
    eps, T, x, kv = c["norm"]["eps"], len(tokens), w["embed"][tokens], {}
    norm = lambda x, g: torch.nn.functional.layer_norm(x, x.shape[-1:], None, None, eps) * g
    for i, layer in enumerate(c["layers"]):
        m, s = {k[len(f"l{i}.mix."):]: v for k, v in w.items() if k.startswith(f"l{i}.mix.")}, layer["mixer"]
        h = norm(x, w[f"l{i}.norm1"])
        if layer["type"] == "mamba2":
            H, P, N = s["heads"], s["vdim"], s["state"]
            z, u, dt = (h @ m["in"].T).split([H * P, H * P + 2 * N, H], 1)
            u = torch.nn.functional.silu(convolve(u, m["conv"], m["conv.b"]))
            v, dt = u[:, :H * P].reshape(T, H, P), torch.nn.functional.softplus(dt + m["dt_bias"])
            B, C = (t[:, None].expand(T, H, N) for t in u[:, H * P:].split(N, 1))
            y = decayed_sums(C, B, v * dt[..., None], -torch.exp(m["A_log"]) * dt) + m["D"][:, None] * v
            y = (rms(y.reshape(T, H * P) * torch.nn.functional.silu(z), eps) * m["norm"]) @ m["o"].T
        elif layer["type"] == "retention":
            H, dim = s["heads"], s["dim"]
            q, k, v = ((h @ m[n].T).reshape(T, H, dim) for n in "qkv")
            q, k = rotate(q, s["rot"]["base"]), rotate(k, s["rot"]["base"]) * dim ** -0.5
            o = decayed_sums(q, k, v, torch.tensor(s["decay"], dtype=torch.float64, device="cuda").log().expand(T, H))
            y = (rms(o, eps).reshape(T, -1) * torch.nn.functional.silu(h @ m["g"].T)) @ m["o"].T
        else:
            if "kv_from" not in s:
                kv[i] = ((rms(h @ m["k"].T, eps) * m["k.norm"]).reshape(T, s["kv_heads"], -1), (h @ m["v"].T).reshape(T, s["kv_heads"], -1))
            q = (rms(h @ m["q"].T, eps) * m["q.norm"]).reshape(T, s["heads"], -1)
            o = attend(q, *kv[s.get("kv_from", i)], s["scale"], s["mask"]["size"])
            y = (o * torch.sigmoid(h @ m["g"].T)[..., None]).reshape(T, -1) @ m["o"].T
        m, limit = {k[len(f"l{i}.mlp."):]: v for k, v in w.items() if k.startswith(f"l{i}.mlp.")}, layer["mlp"]["limit"]
        g = (h @ m["gate"].T + m["gate.b"]).clamp(max=limit)
        up = (h @ m["up"].T + m["up.b"]).clamp(-limit, limit)
        x = x + y + (g * torch.sigmoid(1.702 * g) * (up + 1.0)) @ m["down"].T + m["down.b"]
    return norm(x, w["final.norm"])


@torch.no_grad()
def exact(case, seed):
    w, c, lengths, rows = read_weights(model_folder(case["model"])), MODELS[case["model"]][0], prompt_lengths(case), []
    for n, tokens in zip(lengths, tokens_of(case, seed)):
        t = torch.tensor(tokens, device="cuda")
        if case["model"] == "tupalorn":
            z = tupalorn_hidden(w, c, t)[0 if case["score"] else n - 1:] @ w["embed"].T
            rows.append(c["logit_softcap"] * torch.tanh(z / c["logit_softcap"]))
        else:
            rows.append(lfm2_hidden(w, c, t)[0 if case["score"] else n - 1:] @ w["model.embed_tokens.weight"].T)
    logits = torch.cat(rows)
    return {"logits": logits} if not case["sample"] else {"logits": logits, "tokens": None}
