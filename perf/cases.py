"""The work that users of this library have it do, as cases that can be timed and checked.

A case is one request as a program makes it: prompts enter a loaded model's cache in one step, the first tokens are
chosen, further tokens are decoded one step at a time (forward, choice on the device, the chosen ids read back), and the
slots are given back.  It goes through the public entry points that `LLM.generate` itself is made of: `Context.acquire`,
`forward_batch`, `decode_and_sample`, `release` and `DeviceSampler.sample`.  The tokens that are fed come from the seed
and are not the chosen ones: bfloat16 logits of random weights have near-ties, and two correct implementations that
fed their own choices back would soon compute different sequences.  The outputs are the logits of every step, and in
float32 also the ids.

Every size is one of the repository's presets (`measure.PRESETS`) with random weights, written once per machine.  A loaded
model and its context live as long as the process asks for the same one: requests come and go, the model stays.

The architectures left out share their kernels with the ones here, but choose experts by scores: in bfloat16 two correct
implementations send a few tokens to different experts, and their logits cannot be compared.  Betepel chooses experts by
the token's id.
"""
from __future__ import annotations

import functools
import json
import math
import os
import random
import struct
from typing import Any, Dict, List

import torch
import torch.nn.functional as F

import mini_llama_cpp_release_b200 as ml
from mini_llama_cpp_release_b200 import measure
from mini_llama_cpp_release_b200.sampling import DeviceSampler, SamplingParams


def _case(preset: str, layers: int, batch: int, prompt: int, new: int, name: str = "", **more: Any) -> Dict[str, Any]:
    """`prompt`: tokens of a prompt; with `ragged`, of the longest one.  `new`: tokens chosen per prompt, the first from
    the prompt's own step."""
    c: Dict[str, Any] = dict(preset=preset, layers=layers, dtype="bfloat16", batch=batch, prompt=prompt, new=new,
                             ragged=False, temperature=0.0, top_k=0)
    c.update(more)
    return dict(c, name=name) if name else c


def listed() -> List[Dict[str, Any]]:
    return [
        # the first token of an answer to a short question: one small step, its launches and its latency
        _case("qwen2-0.5b", 24, 1, 23, 1, "first token, 23-token prompt"),
        # one user's chat answer: a short prompt, then single tokens one after the other
        _case("qwen2-0.5b", 24, 1, 61, 64, "answer, batch 1"),
        # the library's headline workload: eight long prompts, each continued
        _case("qwen2-0.5b", 24, 8, 2048, 64, "answers, batch 8, 2048-token prompts"),
        # a server's full batch of short requests of unequal length, sampled
        _case("qwen2-0.5b", 24, 64, 384, 24, "answers, batch 64, ragged, top-k", ragged=True, temperature=0.8, top_k=40),
        # reading one document: a single long step
        _case("qwen2-0.5b", 24, 1, 2048, 1, "prompt of 2048"),
        # reading a long document of an odd length
        _case("qwen2-0.5b", 24, 1, 8191, 1, "prompt of 8191"),
        # the 16 ragged prompts of the benchmark's second configuration
        _case("qwen2-1.5b", 28, 16, 2048, 24, "1.5b answers, batch 16, ragged", ragged=True),
        # layers of the largest preset's width (four of its 28, so that the weights are quickly made)
        _case("qwen2-7b", 4, 8, 511, 48, "7b layers, batch 8"),
        # the library's other element type, for users who check another program against it
        _case("qwen2-0.5b", 24, 3, 100, 16, "float32, batch 3, ragged", ragged=True, dtype="float32"),
        # a mixed model: delta-rule layers, and layers of sink attention beside a linear recurrence
        _case("mepolix-w896", 6, 4, 1000, 48, "mepolix answers, batch 4"),
        # a mixed model: differential and windowed attention, two linear memories, experts by token id; mostly reading
        _case("betepel-w1536", 6, 3, 1500, 1, "betepel prompts, ragged", ragged=True),
        # the same, mostly answering
        _case("betepel-w1536", 6, 8, 120, 48, "betepel answers, batch 8"),
    ]


def _spread(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> Dict[str, Any]:
    preset, layers, most = rng.choice([("qwen2-0.5b", 24, 16384)] * 4 + [("qwen2-1.5b", 28, 12000), ("qwen2-7b", 4, 6000),
                                      ("mepolix-w896", 6, 6000), ("betepel-w1536", 6, 6000)])
    more: Dict[str, Any] = {}
    batch = _spread(rng, 1, 64)
    if preset == "qwen2-0.5b" and rng.random() < 0.2:
        most, batch, more["dtype"] = 600, min(batch, 8), "float32"
    elif rng.random() < 0.3:
        more.update(temperature=0.8, top_k=rng.choice([0, 40]))
    prompt = _spread(rng, 2, min(8192 if batch == 1 else 2048, max(2, most // batch)))
    new = 1 if rng.random() < 0.3 else rng.randint(2, 64)
    if new > 1 and batch > 8:
        new = rng.randint(2, 24)
    return _case(preset, layers, batch, prompt, new, ragged=batch > 1 and rng.random() < 0.6, **more)


# --------------------------------------------------------------------------- what a program has before the call

def _raw(case: Dict[str, Any]) -> Dict[str, Any]:
    raw = dict(measure.PRESETS[case["preset"]])
    if "layers" in raw:
        raw["layers"] = raw["layers"][: case["layers"]]
    else:
        raw["num_hidden_layers"] = case["layers"]
    return raw


def _lengths(case: Dict[str, Any]) -> List[int]:
    if not case["ragged"]:
        return [case["prompt"]] * case["batch"]
    rng = random.Random(case["prompt"] * 1000 + case["batch"])
    return [case["prompt"]] + [rng.randint(1, case["prompt"]) for _ in range(case["batch"] - 1)]


def _tokens(case: Dict[str, Any], seed: int) -> List[List[int]]:
    """For each sequence its prompt and the tokens fed after it; of unequal lengths, another order for another seed."""
    rng = random.Random(seed)
    lengths = _lengths(case)
    rng.shuffle(lengths)
    vocab = measure.PRESETS[case["preset"]].get("vocab_size") or measure.PRESETS[case["preset"]]["vocab"]
    return [[rng.randrange(vocab) for _ in range(n + case["new"] - 1)] for n in lengths]


def _folder(case: Dict[str, Any]) -> str:
    return measure.random_model_folder(_raw(case), tag=f"cases_{case['preset']}_L{case['layers']}")


@functools.lru_cache(maxsize=1)
def _model(preset: str, layers: int, dtype: str) -> Any:
    return ml.load(_folder(dict(preset=preset, layers=layers)), dtype=dtype, max_tokens=64, max_seqs=1).model


@functools.lru_cache(maxsize=1)
def _loaded(preset: str, layers: int, dtype: str, batch: int, per_seq: int) -> Any:
    pages = (per_seq + 63) // 64
    return ml.LLM(_model(preset, layers, dtype), max_tokens=batch * pages * 64, max_seqs=batch)


def prepare(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    llm = _loaded(case["preset"], case["layers"], case["dtype"], case["batch"], case["prompt"] + case["new"])
    n_fed = case["new"] - 1
    rows = _tokens(case, seed)
    return {
        "llm": llm,
        "prompts": [r[: len(r) - n_fed] for r in rows],
        "fed": [[r[len(r) - n_fed + i] for r in rows] for i in range(n_fed)],
        "sampler": DeviceSampler(SamplingParams(case["temperature"], case["top_k"], seed), llm.model.runtime.device),
        "with_ids": case["dtype"] == "float32",
    }


def run(state: Dict[str, Any]) -> Dict[str, Any]:
    ctx, prompts, sampler = state["llm"].context, state["prompts"], state["sampler"]
    ids = list(range(len(prompts)))
    slots = [ctx.acquire() for _ in prompts]
    try:
        logits = ctx.forward_batch(ml.MiniBatch.prefill(slots, prompts))
        chosen = [sampler.sample(logits, ids, [len(p) for p in prompts])]
        out = logits.new_empty(1 + len(state["fed"]), *logits.shape)
        out[0].copy_(logits)
        for i, fed in enumerate(state["fed"]):
            picked, logits = ctx.decode_and_sample(slots, fed, sampler, ids)
            out[i + 1].copy_(logits)
            chosen.append(picked)
    finally:
        for s in slots:
            ctx.release(s)
    return {"logits": out, "ids": torch.tensor(chosen)} if state["with_ids"] else {"logits": out}


# --------------------------------------------------------------------------- what a pass cannot do without

def _weights(raw: Dict[str, Any]):
    """Per layer: (elements every token is multiplied by, elements a step reads, attention heads, entries of a query and a
    value together, window or None, elements of key and value a token leaves, elements of fixed state)."""
    if "layers" not in raw:
        d, ff, H, G, hd = (raw[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
        w = (H + 2 * G) * hd * d + H * hd * d + 3 * ff * d
        return [(w, w, H, 2 * hd, None, 2 * G * hd, 0)] * raw["num_hidden_layers"], d, raw["vocab_size"]
    d, out = raw["width"], []

    def attention(m):
        H, G, hd, dv, maps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], 2 if "diff" in m else 1
        own = "kv_from" not in m
        w = d * (maps * H * hd + H * dv + (own * G * (maps * hd + dv)) + (H if "diff" in m else 0))
        return w, H * maps, hd + dv, (m.get("mask") or {}).get("size"), own * G * (maps * hd + dv)

    for layer in raw["layers"]:
        m, ff = layer["mixer"], layer.get("mlp")
        H_att, entries, window, kv, state = 0, 0, None, 0, 0
        if layer["type"] == "delta":
            H, G, hd, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            w, state = d * (2 * G * hd + 3 * H * dv + 2 * H), H * hd * dv
        elif layer["type"] == "mlstm":
            H, hd, dv = m["heads"], m["dim"], m["vdim"]
            w, state = d * (2 * H * hd + 3 * H * dv + 2 * H), H * hd * dv
        elif layer["type"] == "attention":
            w, H_att, entries, window, kv = attention(m)
        else:
            w, H_att, entries, window, kv = attention(m["left"])
            r = m["right"]
            if "decay" in r:
                w, state = w + d * (2 * r["heads"] * r["dim"] + 3 * r["heads"] * r["vdim"]), r["heads"] * r["dim"] * r["vdim"]
            else:
                w, state = w + 3 * d * r["width"] + 2 * r["width"] ** 2 // r["blocks"], r["width"]
        read = w
        if ff is not None and ff["kind"] == "dense":
            w, read = w + 3 * ff["ff"] * d, read + 3 * ff["ff"] * d
        elif ff is not None:
            one, shared = 3 * ff["expert"]["ff"] * d, 3 * ff["shared"]["ff"] * d
            w, read = w + one * ff["router"]["top"] + shared, read + one * ff["router"]["experts"] + shared
        out.append((w, read, H_att, entries, window, kv, state))
    return out, d, raw["vocab"]


def work(case: Dict[str, Any]) -> Dict[str, float]:
    layers, d, vocab = _weights(_raw(case))
    lengths, steps = _lengths(case), case["new"]
    size = 4 if case["dtype"] == "float32" else 2
    tokens = sum(lengths)
    n_bytes = float(steps) * (sum(x[1] for x in layers) * size + vocab * d * size + len(lengths) * vocab * 4)
    flops = 2.0 * vocab * d * len(lengths) * steps
    for w, _, H, entries, window, kv, state in layers:
        flops += 2.0 * w * (tokens + len(lengths) * (steps - 1)) + 4.0 * state * (tokens + len(lengths) * (steps - 1))
        n_bytes += size * kv * tokens + 8.0 * state * len(lengths) * steps
        for n in lengths:
            w_n = min(window or n, n)
            flops += 2.0 * H * entries * (n * w_n - w_n * w_n / 2)
            for s in range(1, steps):
                seen = min(window or n + s, n + s)
                flops += 2.0 * H * entries * seen
                n_bytes += size * kv * seen
    return {"bytes": n_bytes, "flops": flops}


def tolerance(case: Dict[str, Any]) -> Dict[str, float]:
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-4, "differ": 0.01}
    return {"rel": 0.03, "max": 0.3}


# --------------------------------------------------------------------------- the same in 64 bits

def _read_weights(folder: str) -> Dict[str, torch.Tensor]:
    """model.safetensors on the GPU: floating tensors in 64 bits."""
    path = os.path.join(folder, "model.safetensors")
    with open(path, "rb") as f:
        n = struct.unpack("<Q", f.read(8))[0]
        head = json.loads(f.read(n))
    data = torch.from_file(path, shared=False, size=os.path.getsize(path), dtype=torch.uint8)[8 + n:]
    kinds = {"BF16": torch.bfloat16, "F32": torch.float32, "I32": torch.int32}
    out = {}
    for name, t in head.items():
        if name != "__metadata__":
            lo, hi = t["data_offsets"]
            v = data[lo:hi].cuda().view(kinds[t["dtype"]]).reshape(t["shape"])
            out[name] = v.double() if v.is_floating_point() else v
    return out


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, g, eps):
    return _unit(x - x.mean(-1, keepdim=True), eps) * g


def _swiglu(x, w, p):
    return (F.silu(x @ w[p + "gate"].T) * (x @ w[p + "up"].T)) @ w[p + "down"].T


def _turn(x, rot):
    """x [T, heads, d]: the first `dims` entries of each head, in pairs (i, i + dims/2)."""
    dims, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    f, m = base ** (-2.0 * i / dims), 1.0
    if sc and "fast" in sc:           # stretched by a ramp over the pairs
        def at(turns):
            return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, m = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    elif sc:                          # stretched by the wavelength
        s = ((sc["original"] * f / (2.0 * math.pi) - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)
        f = (1.0 - s) * f / sc["factor"] + s * f
    # angles are defined as float32 products of position and frequency
    a = (torch.arange(len(x), device=x.device).float()[:, None] * f.float()).double()[:, None]
    c, s = torch.cos(a) * m, torch.sin(a) * m
    u, v = x[..., : dims // 2], x[..., dims // 2: dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _attend(q, k, v, scale, mask=None, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv], causal."""
    T, H, rep = len(q), q.shape[1], q.shape[1] // k.shape[1]
    k, v = (t.repeat_interleave(rep, 1).transpose(0, 1) for t in (k, v))
    out, j = [], torch.arange(T, device=q.device)
    for lo in range(0, T, 1024):
        i = j[lo: lo + 1024, None]
        ok = j <= i
        if mask:
            ok = ok & ((i - j < mask["size"]) | (j < (mask.get("keep_first") or 0)))
        s = (q[lo: lo + 1024].transpose(0, 1) @ k.transpose(1, 2) * scale).masked_fill_(~ok, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, s.shape[1], 1)], -1)
        out.append((torch.softmax(s, -1)[..., :T] @ v).transpose(0, 1))
    return torch.cat(out)


def _conv_silu(x, w, b=None, act=True):
    y = F.conv1d(F.pad(x.T, (w.shape[1] - 1, 0)), w[:, None], b, groups=len(w)).T
    return F.silu(y) if act else y


def _qwen2(raw, w, ids):
    H, G, hd, eps = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    rot = {"dims": hd, "base": raw["rope_theta"]}
    x = w["model.embed_tokens.weight"][ids]
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _unit(x, eps) * w[p + "input_layernorm.weight"]
        q, k, v = ((h @ w[f"{p}self_attn.{n}_proj.weight"].T + w[f"{p}self_attn.{n}_proj.bias"]).view(len(x), -1, hd) for n in "qkv")
        x = x + _attend(_turn(q, rot), _turn(k, rot), v, hd ** -0.5).reshape(len(x), H * hd) @ w[p + "self_attn.o_proj.weight"].T
        h = _unit(x, eps) * w[p + "post_attention_layernorm.weight"]
        g, u, dn = (w[f"{p}mlp.{n}_proj.weight"] for n in ("gate", "up", "down"))
        x = x + (F.silu(h @ g.T) * (h @ u.T)) @ dn.T
    head = w["model.embed_tokens.weight" if raw["tie_word_embeddings"] else "lm_head.weight"]
    return lambda rows: (_unit(x[rows], eps) * w["model.norm.weight"]) @ head.T


def _delta(x, w, p, m, eps):
    T, H, G, d, dv = len(x), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k = (_conv_silu(x @ w[p + n].T, w[p + n + ".conv"]).view(T, G, d) for n in "qk")
    v = _conv_silu(x @ w[p + "v"].T, w[p + "v.conv"]).view(T, H, dv)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    beta = torch.sigmoid(x @ w[p + "b"].T)[..., None]
    keep = torch.exp(-torch.exp(w[p + "A_log"]) * F.softplus(x @ w[p + "a"].T + w[p + "dt_bias"]))[..., None, None]
    S, out = x.new_zeros(H, d, dv), []
    for t in range(T):
        S = keep[t] * S
        u = beta[t] * (v[t] - (S * k[t][..., None]).sum(1))
        S = S + k[t][..., None] * u[:, None]
        out.append((S * q[t][..., None]).sum(1))
    y = _unit(torch.stack(out), eps) * w[p + "norm"] * F.silu(x @ w[p + "g"].T).view(T, H, dv)
    return y.reshape(T, -1) @ w[p + "o"].T


def _sink_beside_recurrence(x, w, p, m, eps):
    a, r, T = m["left"], m["right"], len(x)
    q, k, v = ((x @ w[f"{p}left.{n}"].T).view(T, h, e) for n, h, e in (("q", a["heads"], a["dim"]), ("k", a["kv_heads"], a["dim"]), ("v", a["kv_heads"], a["vdim"])))
    q, k = (_turn(_unit(t, eps) * w[f"{p}left.{n}.norm"], a["rot"]) for n, t in (("q", q), ("k", k)))
    left = _attend(q, k, v, a["scale"], sink=w[p + "left.sink"]).reshape(T, -1) @ w[p + "left.o"].T
    p += "right."
    y = F.gelu(x @ w[p + "y"].T + w[p + "y.b"], approximate="tanh")
    u = _conv_silu(x @ w[p + "x"].T + w[p + "x.b"], w[p + "conv"], w[p + "conv.b"], act=False)
    ra, ri = (torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(T, r["blocks"], -1), w[p + n]) + w[p + n + ".b"]).reshape(T, -1) for n in ("ra", "ri"))
    decay = torch.exp(-8.0 * ra * F.softplus(w[p + "lam"]))
    drive, S, out = torch.sqrt(1.0 - decay * decay) * ri * u, torch.zeros_like(u[0]), []
    for t in range(T):
        S = decay[t] * S + drive[t]
        out.append(S)
    return m["left_scale"] * left + m["right_scale"] * ((torch.stack(out) * y) @ w[p + "o"].T)


def _mepolix(raw, w, ids):
    eps, x = raw["norm"]["eps"], w["embed"][ids]
    for i, layer in enumerate(raw["layers"]):
        p = f"l{i}."
        mix = _delta if layer["type"] == "delta" else _sink_beside_recurrence
        x = x + _layer_norm(mix(x, w, p + "mix.", layer["mixer"], eps), w[p + "norm1"], eps)
        x = x + _layer_norm(_swiglu(x, w, p + "mlp."), w[p + "norm2"], eps)
    cap = raw["logit_softcap"]
    return lambda rows: cap * torch.tanh(_layer_norm(x[rows], w["final.norm"], eps) @ w["head"].T / cap)


def _differential(h, w, p, m, eps, kept, i):
    T, H, G, d, dv = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"]

    def maps(n, heads):
        t = (h @ w[p + n].T + w[p + n + ".b"]).view(T, heads, 2, d)
        return [_turn(t[:, :, j], m["rot"]) for j in (0, 1)]
    if "kv_from" not in m:
        kept[i] = (*maps("k", G), (h @ w[p + "v"].T + w[p + "v.b"]).view(T, G, dv))
    k1, k2, v = kept[m.get("kv_from", i)]
    lam = torch.exp((w[p + "lq1"] * w[p + "lk1"]).sum()) - torch.exp((w[p + "lq2"] * w[p + "lk2"]).sum()) + m["diff"]
    a1, a2 = (_attend(q, k, v, m["scale"], m["mask"]) for q, k in zip(maps("q", H), (k1, k2)))
    o = _unit(a1 - lam * a2, eps) * (1.0 - m["diff"]) * torch.sigmoid(h @ w[p + "g"].T)[..., None]
    return o.reshape(T, -1) @ w[p + "o"].T


def _window_beside_decay(h, w, p, m, eps):
    a, r, T = m["left"], m["right"], len(h)
    q, k, v = ((h @ w[f"{p}left.{n}"].T + w[f"{p}left.{n}.b"]).view(T, g, e) for n, g, e in (("q", a["heads"], a["dim"]), ("k", a["kv_heads"], a["dim"]), ("v", a["kv_heads"], a["vdim"])))
    left = _attend(_turn(q, a["rot"]), _turn(k, a["rot"]), v, a["scale"], a["mask"]).reshape(T, -1) @ w[p + "left.o"].T
    p += "right."
    q, k, v = (F.silu(h @ w[p + n].T).view(T, r["heads"], -1) for n in "qkv")
    lam = torch.tensor(r["decay"], dtype=h.dtype, device=h.device)[:, None, None]
    S, out = h.new_zeros(r["heads"], r["dim"], r["vdim"]), []
    for t in range(T):
        S = lam * S + k[t][..., None] * v[t][:, None]
        out.append((S * q[t][..., None]).sum(1).reshape(-1))
    o = _unit(torch.stack(out), eps) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)
    return m["left_scale"] * left + m["right_scale"] * (o @ w[p + "o"].T)


def _matrix_memory(h, w, p, m, eps):
    T, H, cap = len(h), m["heads"], m["gate_cap"]
    q, k, v = ((h @ w[p + n].T).view(T, H, -1) for n in "qkv")
    q = q * m["dim"] ** -0.5
    gi, gf = (cap * torch.tanh((h @ w[p + n].T + w[p + n + ".b"]) / cap) for n in "if")
    gf = F.logsigmoid(gf)
    S, n, top, out = h.new_zeros(H, m["dim"], m["vdim"]), h.new_zeros(H, m["dim"]), h.new_zeros(H), []
    for t in range(T):
        new = torch.maximum(gf[t] + top, gi[t])
        keep, take, top = torch.exp(gf[t] + top - new)[:, None], torch.exp(gi[t] - new)[:, None], new
        S = keep[..., None] * S + (take * k[t])[..., None] * v[t][:, None]
        n = keep * n + take * k[t]
        out.append((S * q[t][..., None]).sum(1) / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6)[:, None])
    o = _unit(torch.stack(out), eps).reshape(T, -1) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)
    return o @ w[p + "o"].T


def _betepel(raw, w, ids):
    eps, kept = raw["norm"]["eps"], {}
    x = _unit(w["embed"][ids], eps) * (1.0 + w["embed.norm"])
    for i, layer in enumerate(raw["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        h = _unit(x, eps) * (1.0 + w[p + "norm1"])
        if layer["type"] == "attention":
            y = _differential(h, w, p + "mix.", m, eps, kept, i)
        else:
            y = (_window_beside_decay if layer["type"] == "parallel" else _matrix_memory)(h, w, p + "mix.", m, eps)
        h = _unit(x, eps) * (1.0 + w[p + "norm2"])
        y = y + _swiglu(h, w, p + "mlp.shared.")
        table = w[p + "mlp.table"][ids]
        for e in range(mlp["router"]["experts"]):
            rows, _ = torch.where(table == e)
            y[rows] += _swiglu(h[rows], w, f"{p}mlp.e{e}.") / mlp["router"]["top"]
        x = x + y
    return lambda rows: _unit(x[rows], eps) * (1.0 + w["final.norm"]) @ w["embed"].T * raw["logit_scale"]


def exact(case: Dict[str, Any], seed: int) -> Any:
    """The logits by whole sequences in 64 bits, without a cache."""
    raw, w = _raw(case), _read_weights(_folder(case))
    forward = {"qwen2": _qwen2, "mepolix": _mepolix, "betepel": _betepel}[case["preset"].split("-")[0]]
    n_fed, rows = case["new"] - 1, []
    for ids in _tokens(case, seed):
        logits = forward(raw, w, torch.tensor(ids, device="cuda"))
        rows.append(logits(slice(len(ids) - n_fed - 1, len(ids))))
    out = torch.stack(rows, 1)
    if case["dtype"] == "float32" and case["temperature"] == 0.0:
        return {"logits": out, "ids": out.argmax(-1).cpu()}
    return {"logits": out, "ids": None} if case["dtype"] == "float32" else {"logits": out}
