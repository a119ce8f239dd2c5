"""What the speed of this framework is measured on: requests as its users send them.

A case is a batch of prompts that start together and then decode a given number of tokens, through the engine's own
calls (`take_slot`, `step`, `sample_async`, `give_back_slot`), as `Engine.generate` makes them.  The tokens that are fed
back are given, not the sampled ones, so that one close call between two tokens does not change everything after it;
sampling itself runs in every step.  Weights are random (N(0, 0.02)), prompts uniform random token ids.

Keys of a case: model (a name of MODELS), dtype, batch, shortest / longest (prompt lengths, spread evenly between the
two), steps (decode steps after the prompt step), temperature and top_p of the sampling.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from odin_infer_b200 import Engine, Engine_Opts, SamplingParams, StepEntry
from odin_infer_b200.config import config_from_dict
from odin_infer_b200.sampling import SequenceSampler
from odin_infer_b200.weights import model_param_specs, random_weights

F64 = torch.float64


# ---------------------------------------------------------------------------------------------------------------
# The models: the Qwen3 sizes that the framework is quoted on, and two of its further architectures at the sizes of
# its own benchmark
# ---------------------------------------------------------------------------------------------------------------
def _qwen3(hidden, inner, layers, heads, kv, head_dim, vocab, theta, eps, tied):
    return dict(architectures=["Qwen3ForCausalLM"], hidden_size=hidden, intermediate_size=inner, num_hidden_layers=layers,
                num_attention_heads=heads, num_key_value_heads=kv, head_dim=head_dim, vocab_size=vocab, rope_theta=theta,
                rms_norm_eps=eps, tie_word_embeddings=tied, max_position_embeddings=40960)


def _nufupel():
    base = {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024}}
    rot = {"dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
    moe = {"kind": "moe", "expert": {"ff": 768}, "router": {"experts": 32, "top": 4}, "shared": {"ff": 1536}}
    layers = []
    for i in range(8):
        if i % 4 == 0:
            layers.append({"type": "attention_2", "mixer": dict(base, rot=rot), "mlp": {"kind": "dense", "ff": 4608} if i == 0 else moe})
        elif i % 4 == 1:
            layers.append({"type": "attention", "mixer": dict(base, mask={"size": 512}), "mlp": moe})
        else:
            layers.append(dict(layers[i - i % 4 + 1], weights_of=i - i % 4 + 1))
    return {"architecture": "Nufupel", "vocab": 32768, "width": 2048, "norm": {"eps": 1e-6},
            "embedding": {"scale": 2048.0 ** 0.5}, "logit_softcap": 30.0, "layers": layers}


def _bafilorn():
    lat = {"heads": 16, "dim": 64, "rot_dim": 64, "vdim": 64, "q_rank": 512, "kv_rank": 64, "scale": 128 ** -0.5,
           "rot": {"dims": 64, "base": 500000.0}}
    lig = {"heads": 16, "dim": 128, "vdim": 128, "decay": [math.exp(-1.0 / (8.0 * 2.0 ** (8.0 * i / 15))) for i in range(16)]}
    par = {"left": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                    "rot": {"dims": 64, "base": 500000.0,
                            "scaling": {"factor": 8.0, "original": 4096, "fast": 24.0, "slow": 1.5}}},
           "right": {"width": 2048, "blocks": 8, "conv": 3}}
    cycle = [("lightning", lig), ("parallel", par), ("latent_attention", lat), ("parallel", par)]
    layers = [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": 6144}} for t, m in (cycle[i % 4] for i in range(8))]
    return {"architecture": "Bafilorn", "vocab": 32768, "width": 2048, "streams": 4, "norm": {"eps": 1e-5},
            "embedding": {"scale": 1.5, "bigram": {"buckets": 99991, "mul_prev": 131, "mul_cur": 31}}, "layers": layers}


MODELS = {
    "tiny-a": _qwen3(64, 128, 2, 4, 2, 16, 256, 1e4, 1e-6, True),
    "tiny-b": _qwen3(96, 224, 3, 6, 2, 32, 384, 1e6, 1e-5, False),
    "qwen3-1.7b": _qwen3(2048, 6144, 28, 16, 8, 128, 151936, 1e6, 1e-6, True),
    "qwen3-8b": _qwen3(4096, 12288, 36, 32, 8, 128, 151936, 1e6, 1e-6, False),
    "nufupel": _nufupel(),
    "bafilorn": _bafilorn(),
}


def _case(model, dtype, batch, shortest, longest, steps, temperature=0.0, top_p=1.0, name=None):
    case = dict(model=model, dtype=dtype, batch=batch, shortest=shortest, longest=longest, steps=steps,
                temperature=temperature, top_p=top_p)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest calls there are: the tiny model in true 32-bit, as a user checks an installation or a port of
        # their own weights against it; launches and host time are all of it
        _case("tiny-a", "float32", 3, 5, 17, 8, name="tiny_greedy_fp32"),
        # the same with drawn tokens: temperature and top-p in every step
        _case("tiny-b", "float32", 4, 1, 40, 12, temperature=0.8, top_p=0.95, name="tiny_sampled_fp32"),
        # a small model answering one short question: latency
        _case("qwen3-1.7b", "bfloat16", 1, 37, 37, 24, name="small_model_one_question"),
        # one chat at the headline size: decoding bound by reading the weights
        _case("qwen3-8b", "bfloat16", 1, 512, 512, 32, name="chat_one"),
        # the headline benchmark: eight sequences with 512-token prompts
        _case("qwen3-8b", "bfloat16", 8, 512, 512, 32, name="chat_eight"),
        # a full server: 64 unequal prompts, then decoding
        _case("qwen3-8b", "bfloat16", 64, 16, 241, 32, name="server_sixty_four"),
        # reading one document: the headline prompt size, no decoding
        _case("qwen3-8b", "bfloat16", 1, 2048, 2048, 0, name="prompt_2048"),
        # a long document and the start of an answer about it
        _case("qwen3-8b", "bfloat16", 1, 12001, 12001, 8, name="long_document"),
        # a batch job of unequal documents on the small model
        _case("qwen3-1.7b", "bfloat16", 64, 16, 2048, 24, name="batch_of_documents"),
        # the true 32-bit path on a real size: reference logits and tokens for some prompts
        _case("qwen3-1.7b", "float32", 4, 61, 400, 8, name="reference_logits_fp32"),
        # experts, windows and sinks: a handful of chats
        _case("nufupel", "bfloat16", 8, 100, 500, 24, name="experts_chat"),
        # linear attention, latent attention and gated units: a document and an answer
        _case("bafilorn", "bfloat16", 2, 900, 2048, 24, name="recurrences_document"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["tiny", "small", "large", "large", "batch", "prompt", "reference", "experts", "recurrences"])
    if kind == "tiny":
        hot = rng.random() < 0.5
        return _case(rng.choice(["tiny-a", "tiny-b"]), "float32", rng.randint(1, 8), rng.randint(1, 16), rng.randint(17, 90),
                     rng.randint(4, 24), temperature=0.8 if hot else 0.0, top_p=0.95 if hot and rng.random() < 0.5 else 1.0)
    if kind == "small":
        a = _log_int(rng, 8, 300)
        return _case("qwen3-1.7b", "bfloat16", _log_int(rng, 1, 16), a, a + _log_int(rng, 1, 300), rng.randint(8, 32))
    if kind == "large":
        batch = _log_int(rng, 1, 96)
        total = _log_int(rng, 64 * batch, max(64 * batch, 10000))   # prompt tokens in all, less than the long document's
        mean = max(8, min(2000, total // batch))
        return _case("qwen3-8b", "bfloat16", batch, max(1, mean // 2), mean + mean // 2, rng.randint(16, 32))
    if kind == "batch":
        batch = _log_int(rng, 8, 64)
        return _case("qwen3-1.7b", "bfloat16", batch, rng.randint(16, 200), _log_int(rng, 300, 2048), rng.randint(8, 24))
    if kind == "prompt":
        n = _log_int(rng, 100, 12001)
        return _case("qwen3-8b", "bfloat16", 1, n, n, rng.choice([0, 0, 8]))
    if kind == "reference":
        a = _log_int(rng, 1, 100)
        return _case("qwen3-1.7b", "float32", rng.randint(1, 6), a, a + _log_int(rng, 10, 250), rng.randint(2, 8))
    if kind == "experts":
        return _case("nufupel", "bfloat16", _log_int(rng, 1, 32), rng.randint(10, 100), _log_int(rng, 128, 700), rng.randint(8, 24))
    return _case("bafilorn", "bfloat16", _log_int(rng, 1, 8), rng.randint(50, 500), _log_int(rng, 600, 2048), rng.randint(8, 24))


# ---------------------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------------------
def _lengths(case):
    a, b, n = case["shortest"], case["longest"], case["batch"]
    return [a + ((b - a) * i) // max(n - 1, 1) for i in range(n)]


def _tokens(case, seed):
    """The prompts, and what is fed after each of them."""
    vocab = _vocab(MODELS[case["model"]])
    rng = np.random.default_rng(seed)
    lengths = _lengths(case)
    lengths = [lengths[i] for i in rng.permutation(len(lengths))]
    prompts = [rng.integers(0, vocab, n).tolist() for n in lengths]
    feed = rng.integers(0, vocab, (case["steps"], case["batch"])).tolist()
    return prompts, feed


def _vocab(raw):
    return raw.get("vocab_size") or raw["vocab"]


def prepare(case, seed):
    """The loaded model with its cache, the prompts and the sampling settings."""
    raw = MODELS[case["model"]]
    prompts, feed = _tokens(case, seed)
    need = [(len(p) + case["steps"] + 63) // 64 * 64 for p in prompts]
    engine = Engine.random(config_from_dict(raw), seed, Engine_Opts(
        max_ctx=max(4096, max(need)), max_tokens=sum(need), max_batch=case["batch"], dtype=case["dtype"], verbose=False))
    return dict(engine=engine, prompts=prompts, feed=feed,
                params=SamplingParams(temperature=case["temperature"], top_p=case["top_p"], seed=seed))


def run(state):
    """The prompts in one step, then one token of every sequence per step; every step's tokens are sampled."""
    engine, prompts, params = state["engine"], state["prompts"], state["params"]
    samplers = [SequenceSampler(params, i, p) for i, p in enumerate(prompts)]
    slots = [engine.take_slot() for _ in prompts]
    try:
        logits = engine.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, prompts)])
        out = {"prompt_logits": logits}
        tokens = [engine.sample_async(logits, samplers, params).device_tokens]
        for row in state["feed"]:
            logits = engine.step([StepEntry(s, [t], [0]) for s, t in zip(slots, row)])
            tokens.append(engine.sample_async(logits, samplers, params).device_tokens)
    finally:
        for s in slots:
            engine.give_back_slot(s)
    if state["feed"]:
        out["last_logits"] = logits
    out["tokens"] = torch.stack(tokens)
    return out


# ---------------------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------
def _matrices(raw):
    """(elements of the layers' matrices that every token passes, times layer runs; the experts' part apart: elements of
    one expert, experts per token, experts, runs of expert layers; elements of the head)."""
    if "hidden_size" in raw:
        d, h = raw["hidden_size"], raw["head_dim"]
        q, kv = raw["num_attention_heads"] * h, raw["num_key_value_heads"] * h
        per = d * (q + 2 * kv) + q * d + 3 * d * raw["intermediate_size"]
        return per * raw["num_hidden_layers"], (0, 0, 0, 0), raw["vocab_size"] * d
    d, total, experts = raw["width"], 0, (0, 0, 0, 0)
    for layer in raw["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        if layer["type"] in ("attention", "attention_2"):
            q, kv = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
            total += d * (2 * q + 2 * kv) + (d * q if layer["type"] == "attention" else d * m["heads"])
        elif layer["type"] == "lightning":
            total += 5 * d * m["heads"] * m["dim"]
        elif layer["type"] == "latent_attention":
            H, e, r, v = m["heads"], m["dim"], m["rot_dim"], m["vdim"]
            total += (d * m["q_rank"] + m["q_rank"] * H * (e + r) + d * (m["kv_rank"] + r) + m["kv_rank"] * H * (e + v) + 2 * d * H * v)
        else:
            left, right = m["left"], m["right"]
            q, kv, w = left["heads"] * left["dim"], left["kv_heads"] * left["dim"], right["width"]
            total += 3 * d * q + d * kv + 3 * d * w + 2 * w * w // right["blocks"]
        if f["kind"] == "dense":
            total += (3 if raw["architecture"] == "Nufupel" else 2) * d * f["ff"]
        else:
            total += 3 * d * f["shared"]["ff"] + d * f["router"]["experts"]
            experts = (3 * d * f["expert"]["ff"], f["router"]["top"], f["router"]["experts"], experts[3] + 1)
    return total, experts, raw["vocab"] * d


def _attention(raw):
    """(elements cached per token and layer, multiplications per (token, key)) of every attention layer, with the most keys
    that a token sees."""
    if "hidden_size" in raw:
        h = raw["head_dim"]
        return [(2 * raw["num_key_value_heads"] * h, 2 * raw["num_attention_heads"] * h, 1 << 30)] * raw["num_hidden_layers"]
    out = []
    for layer in raw["layers"]:
        m = layer["mixer"]
        if layer["type"] == "latent_attention":
            out.append((m["kv_rank"] + m["rot_dim"], m["heads"] * (2 * m["kv_rank"] + m["rot_dim"]), 1 << 30))
        elif layer["type"] != "lightning":
            m = m.get("left", m)
            out.append((2 * m["kv_heads"] * m["dim"], 2 * m["heads"] * m["dim"], m["mask"]["size"]))
    return out


def work(case):
    """Per step every matrix that the step uses is read once (of the experts: as many as its tokens choose on average),
    and every cached row that its tokens see; the logits are written."""
    raw, item = MODELS[case["model"]], 4 if case["dtype"] == "float32" else 2
    dense, (expert, top, n_experts, moe_layers), head = _matrices(raw)
    lengths = _lengths(case)
    tokens, batch, steps = sum(lengths), case["batch"], case["steps"]
    nbytes, flops = 0.0, 0.0
    for rows in [tokens] + [batch] * steps:
        touched = n_experts * (1.0 - (1.0 - 1.0 / n_experts) ** (rows * top)) if n_experts else 0.0
        nbytes += item * (dense + head + expert * touched * moe_layers) + 4.0 * batch * _vocab(raw)
        flops += 2.0 * rows * (dense + expert * top * moe_layers) + 2.0 * batch * head
    for cached, mults, most in _attention(raw):
        for n in lengths:
            seen = sum(min(p + 1, most) for p in range(n))
            nbytes += item * cached * n
            for s in range(steps):
                nbytes += item * cached * min(n + s + 1, most)
                seen += min(n + s + 1, most)
            flops += 2.0 * mults * seen
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times the errors against `exact` that were measured: 1e-5 in 32-bit on the 28 layers of the 1.7B size,
    0.037 in bfloat16 on the 36 layers of the 8B size, 0.025 with experts (a router's close calls send a token to another
    one), 0.0033 for the recurrences."""
    if case["dtype"] == "float32":
        return {"rel": 4e-5, "max": 4e-4, "differ": 0.05}
    if case["model"] == "bafilorn":
        return {"rel": 1.5e-2, "max": 0.12, "differ": 0.15}
    return {"rel": 0.1 if case["model"] == "nufupel" else 0.14, "max": 0.9, "differ": 0.3}


# ---------------------------------------------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------------------------------------------
class _Reader:
    """Weights by name, widened when they are asked for."""

    def __init__(self, tensors):
        self.tensors = tensors

    def __getitem__(self, name):
        return self.tensors[name].to(F64)


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu_tanh(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _angles(positions, freq, in_32_bit=True):
    """The angle of a rotation is a 32-bit product by these models' definition, unless they say otherwise."""
    if in_32_bit:
        ang = (positions.astype(np.float32)[:, None] * freq.astype(np.float32)[None, :]).astype(np.float32).astype(np.float64)
    else:
        ang = positions.astype(np.float64)[:, None] * freq[None, :]
    return torch.from_numpy(np.cos(ang)).cuda()[:, None, :], torch.from_numpy(np.sin(ang)).cuda()[:, None, :]


def _rotate(t, cos, sin, pairs=False):
    """t: [rows, heads, dim]; the first 2 * cos.shape[-1] elements of every head turn."""
    half = cos.shape[-1]
    out = t.clone()
    u, v = (t[..., 0:2 * half:2], t[..., 1:2 * half:2]) if pairs else (t[..., :half], t[..., half:2 * half])
    a, b = u * cos - v * sin, v * cos + u * sin
    if pairs:
        out[..., 0:2 * half:2], out[..., 1:2 * half:2] = a, b
    else:
        out[..., :half], out[..., half:2 * half] = a, b
    return out


def _attend(q, k, v, lengths, scale, window=0, chunk=0, sink=None):
    """Causal attention sequence by sequence; q: [rows, H, e], k, v: [rows, G, e]; sink: [H], logits that join the
    softmax's denominator."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=F64, device=q.device)
    r0 = 0
    for n in lengths:
        kk = k[r0:r0 + n].permute(1, 2, 0).unsqueeze(1)                # [G, 1, e, n]
        vv = v[r0:r0 + n].permute(1, 0, 2).unsqueeze(1)                # [G, 1, n, ev]
        j = torch.arange(n, device=q.device)
        rows = max(16, int(4e8 / (8.0 * H * n)))
        for a in range(0, n, rows):
            i = j[a:a + rows]
            qq = q[r0 + a:r0 + a + len(i)].view(len(i), G, H // G, -1).permute(1, 2, 0, 3)
            s = torch.matmul(qq, kk) * scale
            hidden = j[None, :] > i[:, None]
            if window:
                hidden |= i[:, None] - j[None, :] >= window
            if chunk:
                hidden |= i[:, None] // chunk != j[None, :] // chunk
            s.masked_fill_(hidden, -math.inf)
            m = s.amax(dim=-1, keepdim=True)
            if sink is not None:
                extra = sink.view(G, H // G, 1, 1)
                m = torch.maximum(m, extra)
            s.sub_(m).exp_()
            den = s.sum(dim=-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(extra - m)
            o = torch.matmul(s, vv) / den
            out[r0 + a:r0 + a + len(i)] = o.permute(2, 0, 1, 3).reshape(len(i), H, -1)
        r0 += n
    return out


def _positions(lengths):
    return np.concatenate([np.arange(n) for n in lengths])


def _hidden_qwen3(raw, w, ids, lengths):
    eps, h = raw["rms_norm_eps"], raw["head_dim"]
    H, G = raw["num_attention_heads"], raw["num_key_value_heads"]
    i = np.arange(h // 2, dtype=np.float32)
    freq = (np.float32(1.0) / np.power(np.float32(raw["rope_theta"]), i / np.float32(h // 2))).astype(np.float32)
    cos, sin = _angles(_positions(lengths), freq)
    x = w.tensors["model.embed_tokens.weight"][ids].to(F64)
    for layer in range(raw["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        a = _rms(x, w[p + "input_layernorm.weight"], eps)
        q = (a @ w[p + "self_attn.q_proj.weight"].T).view(-1, H, h)
        k = (a @ w[p + "self_attn.k_proj.weight"].T).view(-1, G, h)
        v = (a @ w[p + "self_attn.v_proj.weight"].T).view(-1, G, h)
        q = _rotate(_rms(q, w[p + "self_attn.q_norm.weight"], eps), cos, sin)
        k = _rotate(_rms(k, w[p + "self_attn.k_norm.weight"], eps), cos, sin)
        o = _attend(q, k, v, lengths, h ** -0.5)
        x = x + o.reshape(-1, H * h) @ w[p + "self_attn.o_proj.weight"].T
        a = _rms(x, w[p + "post_attention_layernorm.weight"], eps)
        g = _silu(a @ w[p + "mlp.gate_proj.weight"].T)
        g *= a @ w[p + "mlp.up_proj.weight"].T
        x = x + g @ w[p + "mlp.down_proj.weight"].T
    head = "model.embed_tokens.weight" if raw["tie_word_embeddings"] else "lm_head.weight"
    return lambda rows: _rms(x[rows], w["model.norm.weight"], eps) @ w[head].T


def _stretched(rot):
    st, f = rot["scaling"], rot["base"] ** (-2.0 * np.arange(rot["dims"] // 2) / rot["dims"])
    wave = 2.0 * np.pi / f
    s = (st["original"] / wave - st["low"]) / (st["high"] - st["low"])
    return np.where(wave < st["original"] / st["high"], f, np.where(
        wave > st["original"] / st["low"], f / st["factor"], (1.0 - s) * f / st["factor"] + s * f))


def _hidden_nufupel(raw, w, ids, lengths):
    eps = raw["norm"]["eps"]
    x = w.tensors["embed"][ids].to(F64) * raw["embedding"]["scale"]
    pos = _positions(lengths)

    def gated(h, p, act):
        return (act(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T

    for number, layer in enumerate(raw["layers"]):
        p = f"l{layer.get('weights_of', number)}."
        m, mix = layer["mixer"], p + "mix."
        H, G, e = m["heads"], m["kv_heads"], m["dim"]
        h = _rms(x, 1.0 + w[p + "norm1"], eps)
        q, k, v = ((h @ w[mix + s].T).view(h.shape[0], -1, e) for s in "qkv")
        if layer["type"] == "attention_2":
            cos, sin = _angles(pos, _stretched(m["rot"]))
            q = _rotate(_rms(q, w[mix + "q.norm"], eps), cos, sin)
            k = _rotate(_rms(k, w[mix + "k.norm"], eps), cos, sin)
        o = _attend(q, k, v, lengths, m["scale"], window=m["mask"]["size"], sink=w[mix + "sink"])
        gate = torch.sigmoid(h @ w[mix + "g"].T)
        o = o * (gate[:, :, None] if layer["type"] == "attention_2" else gate.view(-1, H, e))
        update = o.reshape(-1, H * e) @ w[mix + "o"].T
        f, mlp = layer["mlp"], p + "mlp."
        if f["kind"] == "dense":
            update = update + gated(h, mlp, _gelu_tanh)
        else:
            z, chosen = torch.topk(h @ w[mlp + "router"].T + w[mlp + "router.b"], f["router"]["top"], dim=-1)
            share = torch.softmax(z, dim=-1)
            update = update + gated(h, mlp + "shared.", _silu)
            for n in range(f["router"]["experts"]):
                row, place = (chosen == n).nonzero(as_tuple=True)
                update.index_add_(0, row, gated(h[row], f"{mlp}e{n}.", _silu) * share[row, place][:, None])
        x = x + update
    cap = raw["logit_softcap"]
    return lambda rows: cap * torch.tanh(_rms(x[rows], 1.0 + w["final.norm"], eps) @ w["head"].T / cap)


def _ramped(rot):
    st, dims, base = rot["scaling"], rot["dims"], rot["base"]
    f = base ** (-2.0 * np.arange(dims // 2) / dims)

    def pair_of(turns):
        return dims * math.log(st["original"] / (turns * 2.0 * math.pi)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(pair_of(st["fast"])), 0), min(math.ceil(pair_of(st["slow"])), dims - 1)
    r = np.clip((np.arange(dims // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return f / st["factor"] * r + f * (1.0 - r), 0.1 * math.log(st["factor"]) + 1.0


def _hidden_bafilorn(raw, w, ids, lengths):
    eps, pos = raw["norm"]["eps"], _positions(lengths)
    pair = raw["embedding"]["bigram"]
    before = torch.roll(ids, 1)
    rows = (before * pair["mul_prev"] + ids * pair["mul_cur"]) % pair["buckets"]
    rows[torch.from_numpy(pos == 0).cuda()] = pair["buckets"]
    x = w.tensors["embed"][ids].to(F64) * raw["embedding"]["scale"] + w.tensors["bigram"][rows].to(F64)
    X = torch.stack([x] * raw["streams"])
    starts = np.cumsum([0] + list(lengths))

    def read(p):
        return torch.einsum("i,ind->nd", w[p + ".in"], X)

    def join(p, y):
        return torch.einsum("ij,ind->jnd", w[p + ".mix"], X) + w[p + ".out"][:, None, None] * y

    def latent(h, p, m):
        H, e, r, ev, kr = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        cos, sin = _angles(pos, m["rot"]["base"] ** (-2.0 * np.arange(r // 2) / r), in_32_bit=False)
        q = (_rms(h @ w[p + "dq"].T, w[p + "dq.norm"], eps) @ w[p + "uq"].T).view(-1, H, e + r)
        down = h @ w[p + "dkv"].T
        c = _rms(down[:, :kr], w[p + "dkv.norm"], eps)
        k_rot = _rotate(down[:, None, kr:], cos, sin, pairs=True)
        q = torch.cat([q[:, :, :e], _rotate(q[:, :, e:], cos, sin, pairs=True)], dim=2)
        k = torch.cat([(c @ w[p + "uk"].T).view(-1, H, e), k_rot.expand(-1, H, r)], dim=2)
        o = _attend(q, k, (c @ w[p + "uv"].T).view(-1, H, ev), lengths, m["scale"])
        return (o.reshape(-1, H * ev) * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T

    def lightning(h, p, m):
        H, e = m["heads"], m["dim"]
        q, k, v = (_silu(h @ w[p + s].T).view(-1, H, e) for s in "qkv")
        o = torch.empty_like(v)
        log_decay = torch.log(torch.tensor(m["decay"], dtype=F64, device=h.device))
        for a, b in zip(starts[:-1], starts[1:]):
            j = torch.arange(b - a, device=h.device, dtype=F64)
            gap = j[:, None] - j[None, :]
            for head in range(H):
                fade = torch.where(gap >= 0, torch.exp(gap.clamp(min=0) * log_decay[head]), 0.0)
                o[a:b, head] = ((q[a:b, head] @ k[a:b, head].T) * fade) @ v[a:b, head]
        return (_rms(o.reshape(-1, H * e), w[p + "norm"], eps) * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T

    def key_attention(h, p, m):
        H, G, e = m["heads"], m["kv_heads"], m["dim"]
        freq, gain = _ramped(m["rot"])
        cos, sin = (t * gain for t in _angles(pos, freq, in_32_bit=False))
        q = (h @ w[p + "q"].T + w[p + "q.b"]).view(-1, H, e)
        k = (h @ w[p + "k"].T + w[p + "k.b"]).view(-1, G, e)
        o = _attend(_rotate(q, cos, sin), _rotate(k, cos, sin), k, lengths, m["scale"], chunk=m["mask"]["size"],
                    sink=torch.zeros(H, dtype=F64, device=h.device))
        return (o.reshape(-1, H * e) * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T + w[p + "o.b"]

    def unit(h, p, m):
        y = _gelu_tanh(h @ w[p + "y"].T + w[p + "y.b"])
        z = h @ w[p + "x"].T + w[p + "x.b"]
        taps, blocks = w[p + "conv"], m["blocks"]
        n = max(lengths)
        padded = torch.zeros(len(lengths), n + taps.shape[1] - 1, z.shape[1], dtype=F64, device=h.device)
        for s, (a, b) in enumerate(zip(starts[:-1], starts[1:])):
            padded[s, taps.shape[1] - 1:taps.shape[1] - 1 + b - a] = z[a:b]
        u = w[p + "conv.b"] + sum(padded[:, j:j + n] * taps[:, j] for j in range(taps.shape[1]))

        def gate(s):
            parts = torch.einsum("snbm,bom->snbo", u.view(len(lengths), n, blocks, -1), w[p + s])
            return torch.sigmoid(parts + w[p + s + ".b"].view(blocks, -1)).reshape(u.shape)
        log_a = -8.0 * gate("ra") * torch.nn.functional.softplus(w[p + "lam"])
        a, add = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * gate("ri") * u
        S = torch.zeros_like(u[:, 0])
        states = torch.empty_like(u)
        for t in range(n):
            S = torch.addcmul(add[:, t], a[:, t], S)
            states[:, t] = S
        states = torch.cat([states[s, :k] for s, k in enumerate(lengths)])
        return (states * y) @ w[p + "o"].T

    for number, layer in enumerate(raw["layers"]):
        p, m = f"l{number}.", layer["mixer"]
        h = _rms(read(p + "hc1"), 1.0 + w[p + "norm1"], eps)
        if layer["type"] == "lightning":
            y = lightning(h, p + "mix.", m)
        elif layer["type"] == "latent_attention":
            y = latent(h, p + "mix.", m)
        else:
            left, right = key_attention(h, p + "mix.left.", m["left"]), unit(h, p + "mix.right.", m["right"])
            y = 0.5 * (_rms(left, w[p + "mix.left.out"], eps) + _rms(right, w[p + "mix.right.out"], eps))
        X = join(p + "hc1", y)
        h = _rms(read(p + "hc2"), 1.0 + w[p + "norm2"], eps)
        X = join(p + "hc2", torch.relu(h @ w[p + "mlp.up"].T) ** 2 @ w[p + "mlp.down"].T)
    return lambda rows: _rms(X.sum(dim=0)[rows], 1.0 + w["final.norm"], eps) @ w["head"].T


def exact(case, seed):
    """The logits in 64 bits, every sequence whole (its prompt and what is fed after it), and the greedy tokens; drawn
    tokens have no exact value."""
    raw = MODELS[case["model"]]
    prompts, feed = _tokens(case, seed)
    steps = len(feed)
    whole = [p + [row[i] for row in feed] for i, p in enumerate(prompts)]
    lengths = [len(t) for t in whole]
    weights = _Reader(random_weights(model_param_specs(config_from_dict(raw)), seed, torch.bfloat16, "cuda:0"))
    ids = torch.tensor([t for seq in whole for t in seq], dtype=torch.long, device="cuda:0")
    hidden = {"Qwen3ForCausalLM": _hidden_qwen3, "Nufupel": _hidden_nufupel, "Bafilorn": _hidden_bafilorn}
    logits_of = hidden[raw.get("architecture") or raw["architectures"][0]](raw, weights, ids, lengths)
    ends = torch.from_numpy(np.cumsum(lengths) - 1).cuda()
    out, tokens = {"prompt_logits": logits_of(ends - steps)}, []
    for s in range(steps + 1):
        logits = logits_of(ends - steps + s)
        tokens.append(logits.argmax(dim=-1).to(torch.int32))
    if steps:
        out["last_logits"] = logits
    out["tokens"] = torch.stack(tokens) if case["temperature"] == 0.0 else None
    return out


if __name__ == "__main__":
    for c in listed() + [draw(random.Random(s)) for s in range(12)]:
        w = work(c)
        print(f"{c.get('name', 'drawn'):28s} {w['bytes'] / 1e9:9.2f} GB {w['flops'] / 1e12:9.3f} TFLOP  {c}")
