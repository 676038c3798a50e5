"""The work that this framework is measured on: requests to quantised decoders through the session calls, one decoder layer through the
operator calls, and layer-list models through the session and the step calls.

Sizes are those of ``forge_llm_b200.configs.CONFIGS`` and of the layer-list models that the benchmark builds; deep or wide models keep their
layers' shapes and have fewer of them.  Weights and token ids are drawn on the GPU from the seed.  Embeddings have unit variance and the
head's row of a token's successor points along the token's embedding, so that, as in a trained model, the most likely token stands out
and greedy decoding does not hang on the last bits of a logit."""
from __future__ import annotations

import ctypes as C
import json
import math
import os
import random
import shutil
import struct
import tempfile

import numpy as np
import torch

from forge_llm_b200 import configs, synth
from forge_llm_b200._lib import check, lib
from forge_llm_b200.engine import Engine
from forge_llm_b200.runtime import Model

Q4_K, Q6_K = configs.Q4_K, configs.Q6_K


# ------------------------------------------------------------------------------------------------------------------------ cases
def _request(shape, layers, batch, shortest, longest, new, quant=0):
    """Prompts of ``shortest`` .. ``longest`` tokens, then ``new`` greedy tokens for all sequences together (0: the prompts alone)."""
    return {"path": "request", "shape": shape, "layers": layers, "quant": quant, "batch": batch, "shortest": shortest, "longest": longest, "new": new}


def _layer(shape, rows, context):
    """One decoder layer over ``rows`` new positions behind ``context`` cached ones, operator by operator."""
    return {"path": "layer", "shape": shape, "rows": rows, "context": context}


def _stack(design, width, layers, heads, ff, batch, shortest, longest, new, budget):
    return {"path": "stack", "design": design, "width": width, "layers": layers, "heads": heads, "ff": ff, "batch": batch, "shortest": shortest,
            "longest": longest, "new": new, "budget": budget}


def listed():
    return [
        # the smallest calls: a generated program that calls the operators one after another to decode a token of the smallest model
        dict(_layer("c1", 1, 99), name="layer_small_token"),
        # the same program on the prompt of a 1B model
        dict(_layer("c2", 1000, 0), name="layer_prompt_1k"),
        # a short chat with the smallest model (Q8_0, three key heads): launches and latency
        dict(_request("c1", 30, 1, 100, 100, 64), name="chat_135m_q8"),
        # the benchmark's request: a 1501-token prompt and 128 tokens from a 1B model in Q4_0
        dict(_request("c2", 16, 1, 1501, 1501, 128), name="chat_1b_q4"),
        # the same model reading: a long prompt whose next token alone is wanted (classification, scoring, time to the first token)
        dict(_request("c2", 16, 1, 2501, 2501, 0), name="prompt_1b_q4"),
        # a server with 64 requests in flight on a 0.5B model with biases, ragged prompts
        dict(_request("c3", 24, 64, 64, 2501, 32), name="serve64_05b_q8"),
        # a server with 16 requests on a multi-head model with heads of 96, decoding over full caches
        dict(_request("c4", 8, 16, 300, 900, 96), name="serve16_phi_q8"),
        # eight sequences of a 7B model in Q4_0, 2048-token prompts
        dict(_request("c5", 8, 8, 2048, 2048, 64), name="serve8_7b_q4"),
        # K-quants as files of the Q4_K_M kind mix them; the prompt goes token by token, as is the default
        dict(_request("c2", 4, 1, 48, 48, 80, "q4_k_m"), name="chat_1b_q4km"),
        # a layer-list model in bfloat16 with latent attention: a long prompt, then tokens chosen by the caller from the logits
        dict(_stack("bolenex", 2048, 4, 16, 8192, 1, 2048, 2048, 32, 2048), name="bolenex_chat"),
        # a layer-list model served by steps that mix portions of prompts and single tokens: windows, gated linear attention, experts, a loop
        dict(_stack("mokatar", 2048, 8, 16, 8192, 16, 100, 700, 24, 512), name="mokatar_serve16"),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["layer", "request", "request", "request", "request", "stack"])
    if kind == "layer":
        rows = rng.choice([1, spread(8, 1500)])
        return _layer(rng.choice(sorted(configs.CONFIGS)), rows, spread(1, 2000) if rows == 1 else rng.choice([0, spread(1, 500)]))
    if kind == "stack":
        design = rng.choice(["bolenex", "mokatar"])
        batch = rng.choice([1, spread(1, 24)])
        top = spread(100, 2048 if batch == 1 else 700)
        return _stack(design, rng.choice([1024, 2048]), rng.choice([4, 8]), rng.choice([8, 16]), rng.choice([2752, 4096, 8192]), batch, max(1, top // rng.choice([1, 2, 5])), top,
                      spread(8, 40), rng.choice([256, 512, 2048]))
    shape = rng.choice(sorted(configs.CONFIGS))
    quant = rng.choice([0, 0, 0, 4 if configs.CONFIGS[shape]["quant"] == 8 else 8, "q4_k_m" if shape == "c2" else 0])
    if quant == "q4_k_m":
        top = spread(9, 90)
        return _request(shape, rng.randint(2, 4), 1, top, top, spread(8, 80), quant)
    batch = rng.choice([1, spread(2, 8), spread(2, 64)])
    top = spread(9, 2501 if batch <= 8 else 700)
    return _request(shape, rng.randint(2, 8), batch, max(1, top // rng.choice([1, 2, 7])), top, rng.choice([0, spread(8, 96), spread(8, 96)]), quant)


def _lengths(case):
    r = random.Random(case["batch"] * 7919 + case["longest"])
    n = [r.randint(case["shortest"], case["longest"]) for _ in range(case["batch"])]
    n[-1] = case["longest"]
    return n


def _config(case):
    c = dict(configs.CONFIGS[case["shape"]])
    if case["path"] == "request":
        c["num_layers"] = case["layers"]
        c["tied"] = False
        if case["quant"] == "q4_k_m":
            c["quant"] = Q4_K
            c = configs.with_proj_quant(c, v=Q6_K, down=Q6_K, lm_head=Q6_K)
        elif case["quant"]:
            c["quant"] = case["quant"]
    return c


# ---------------------------------------------------------------------------------------------------------------------- weights
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _f16_bytes(x):
    return x.to(torch.float16).contiguous().view(torch.uint8).reshape(-1, 2)


def _scales_q8(x):
    """Scale and inverse of blocks of 32 as a block stores them (f16) and as they round their values (f32)."""
    d = x.abs().amax(1) / 127.0
    return d, torch.where(d > 0, 1.0 / d, torch.zeros_like(d))


def _pack(quant, w):
    """f32 [rows][K] -> the bytes of its blocks, as the formats lay them out."""
    if quant in (8, 4):
        b = w.reshape(-1, 32)
        if quant == 8:
            d, inv = _scales_q8(b)
            q = torch.clamp(torch.round(b * inv[:, None]), -127, 127).to(torch.int8).view(torch.uint8)
        else:
            d = b.gather(1, b.abs().argmax(1, keepdim=True))[:, 0] / -8.0
            inv = torch.where(d != 0, 1.0 / d, torch.zeros_like(d))
            n = torch.clamp(torch.round(b * inv[:, None]) + 8, 0, 15).to(torch.uint8)
            q = n[:, :16] | (n[:, 16:] << 4)
        return torch.cat([_f16_bytes(d), q], 1).reshape(-1)
    if quant == Q4_K:
        s = w.reshape(-1, 8, 32)
        low = torch.clamp(-s.amin(2), min=0)
        step = (s.amax(2) + low) / 15
        d, dmin = (step.amax(1) / 63).to(torch.float16), (low.amax(1) / 63).to(torch.float16)
        sc = torch.clamp(torch.round(step / d.float()[:, None]), 1, 63)
        mn = torch.clamp(torch.round(low / dmin.float()[:, None]), 0, 63)
        q = torch.round((s + (dmin.float()[:, None] * mn)[:, :, None]) / (d.float()[:, None] * sc)[:, :, None])
        q = torch.clamp(q, 0, 15).to(torch.uint8)
        sc, mn = sc.to(torch.uint8), mn.to(torch.uint8)
        scales = torch.cat([sc[:, :4] | ((sc[:, 4:] >> 4) << 6), mn[:, :4] | ((mn[:, 4:] >> 4) << 6), (sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)], 1)
        nib = torch.cat([q[:, 2 * i] | (q[:, 2 * i + 1] << 4) for i in range(4)], 1)
        return torch.cat([d.view(torch.uint8).reshape(-1, 2), dmin.view(torch.uint8).reshape(-1, 2), scales, nib], 1).reshape(-1)
    s = w.reshape(-1, 16, 16)
    step = s.abs().amax(2) / 31
    d = (step.amax(1) / 127).to(torch.float16)
    sc = torch.clamp(torch.round(step / d.float()[:, None]), 1, 127)
    q = (torch.clamp(torch.round(s / (d.float()[:, None] * sc)[:, :, None]), -32, 31) + 32).to(torch.uint8).reshape(-1, 2, 4, 32)
    ql = torch.cat([(q[:, h, i] & 15) | ((q[:, h, i + 2] & 15) << 4) for h in (0, 1) for i in (0, 1)], 1)
    qh = torch.cat([(q[:, h, 0] >> 4) | ((q[:, h, 1] >> 4) << 2) | ((q[:, h, 2] >> 4) << 4) | ((q[:, h, 3] >> 4) << 6) for h in (0, 1)], 1)
    return torch.cat([ql, qh, sc.to(torch.int8).view(torch.uint8), d.view(torch.uint8).reshape(-1, 2)], 1).reshape(-1)


def _unpack(quant, raw, rows):
    """The values of _pack's bytes in float64, [rows][K]."""
    def f16(x):
        return x.contiguous().view(torch.float16).double()

    if quant == 8:
        b = raw.reshape(-1, 34)
        w = b[:, 2:].contiguous().view(torch.int8).double() * f16(b[:, :2])
    elif quant == 4:
        b = raw.reshape(-1, 18)
        w = (torch.cat([b[:, 2:] & 15, b[:, 2:] >> 4], 1).double() - 8) * f16(b[:, :2])
    elif quant == Q4_K:
        b = raw.reshape(-1, 144)
        d, dmin, s = f16(b[:, 0:2]), f16(b[:, 2:4]), b[:, 4:16]
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1).double()
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1).double()
        n = b[:, 16:].reshape(-1, 4, 1, 32)
        q = torch.cat([n & 15, n >> 4], 2).reshape(-1, 8, 32).double()
        w = (d * sc)[:, :, None] * q - (dmin * mn)[:, :, None]
    else:
        b = raw.reshape(-1, 210)
        ql, qh = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 32)
        lo = torch.cat([ql & 15, ql >> 4], 2)
        hi = torch.stack([(qh >> (2 * i)) & 3 for i in range(4)], 2)
        q = (lo | (hi << 4)).reshape(-1, 16, 16).double() - 32
        w = (f16(b[:, 208:]) * b[:, 192:208].contiguous().view(torch.int8).double())[:, :, None] * q
    return w.reshape(rows, -1)


def _successors(seed, vocab):
    return torch.randperm(vocab, generator=_generator(seed + 1), device="cuda")


def _decoder_tensors(c, seed):
    """(name, quant or None, rows, tensor on the GPU) in the order of weights.bin."""
    g = _generator(seed)
    h, hd, ff, V = c["hidden_size"], c["head_dim"], c["intermediate_size"], c["vocab_size"]
    qk, kv = c["num_heads"] * hd, c["num_kv_heads"] * hd
    pq = configs.proj_quants(c)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    embed = normal(V, h)
    yield "embed", None, V, embed
    for i in range(c["num_layers"]):
        yield f"{i}.attn_norm", None, 1, 1 + 0.1 * normal(h)
        for cat, name, rows, k in ((0, "q", qk, h), (1, "k", kv, h), (2, "v", kv, h)):
            yield f"{i}.{name}", pq[cat], rows, _pack(pq[cat], 0.02 * normal(rows, k))
        if c["qkv_bias"]:
            for name, rows in (("qb", qk), ("kb", kv), ("vb", kv)):
                yield f"{i}.{name}", None, 1, 0.02 * normal(rows)
        yield f"{i}.o", pq[3], h, _pack(pq[3], 0.02 * normal(h, qk))
        yield f"{i}.ffn_norm", None, 1, 1 + 0.1 * normal(h)
        for cat, name, rows, k in ((4, "gate", ff, h), (5, "up", ff, h), (6, "down", h, ff)):
            yield f"{i}.{name}", pq[cat], rows, _pack(pq[cat], 0.02 * normal(rows, k))
    yield "norm", None, 1, 1 + 0.1 * normal(h)
    nxt = _successors(seed, V)
    head = torch.empty_like(embed)
    head[nxt] = 0.02 * embed
    head += 0.01 * normal(V, h)
    yield "head", pq[7], V, _pack(pq[7], head)


def _image(c, seed):
    host = torch.empty(synth.weights_bin_size(c), dtype=torch.uint8, pin_memory=True)
    at = 0
    for _, _, _, t in _decoder_tensors(c, seed):
        raw = t.contiguous().view(torch.uint8).reshape(-1)
        host[at:at + raw.numel()].copy_(raw, non_blocking=True)
        at += raw.numel()
    torch.cuda.synchronize()
    return host.numpy()


def _prompts(case, vocab, seed):
    r = np.random.default_rng(seed)
    return [r.integers(0, vocab, n).astype(np.uint32) for n in _lengths(case)]


def _stack_config(case):
    make = {"bolenex": synth.bolenex_config, "mokatar": synth.mokatar_config}[case["design"]]
    return make(case["width"], case["layers"], case["heads"], case["ff"], 32768)


def _stack_tensors(cfg, seed):
    """Matrices N(0, 1 / inputs), factors around their neutral value; everything is a bfloat16 value."""
    g = _generator(seed)
    out = {}
    for name, shape in synth.stack_shapes(cfg).items():
        if name.endswith("alpha"):
            x = torch.full(shape, 0.5, device="cuda")
        elif len(shape) >= 2:
            x = torch.randn(*shape, generator=g, device="cuda") * (1.0 if name in ("embed", "bigram", "loop.step") else shape[1] ** -0.5)
        else:
            around = 0.0 if name.endswith((".b", ".sink")) or (cfg["architecture"] == "Mokatar" and ("norm1" in name or "norm2" in name or name == "final.norm")) else 1.0
            x = around + 0.1 * torch.randn(*shape, generator=g, device="cuda")
        out[name] = x.to(torch.bfloat16)
    return out


def _write_folder(folder, cfg, tensors):
    head, at = {}, 0
    for name, x in tensors.items():
        n = 2 * x.numel()
        head[name] = {"dtype": "BF16", "shape": list(x.shape), "data_offsets": [at, at + n]}
        at += n
    text = json.dumps(head).encode()
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(cfg, f)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(text)) + text)
        f.write(torch.cat([x.reshape(-1) for x in tensors.values()]).view(torch.uint8).cpu().numpy().data)


def _follow_ups(case, vocab, seed):
    """Tokens that the caller appends, [batch][new]."""
    return np.random.default_rng(seed + 2).integers(0, vocab, (case["batch"], case["new"])).astype(np.uint32)


def _plan(case, prompts, follow):
    """Steps of a server: every running request one token, waiting prompts in portions into the rest of the step's budget.  The logits behind
    each prompt and behind each appended token are wanted."""
    prompts, follow = [p.tolist() for p in prompts], follow.tolist()
    fed, made, steps = [0] * len(prompts), [0] * len(prompts), []
    while any(m < case["new"] for m in made):
        left, step = case["budget"], []
        for r, p in enumerate(prompts):
            if fed[r] == len(p) and made[r] < case["new"]:
                step.append((r, [follow[r][made[r]]], [0]))
                made[r] += 1
                left -= 1
        for r, p in enumerate(prompts):
            n = min(left, len(p) - fed[r])
            if n > 0:
                step.append((r, p[fed[r]:fed[r] + n], [n - 1] if fed[r] + n == len(p) else []))
                fed[r] += n
                left -= n
        steps.append(step)
    return steps


def _layer_inputs(case, seed):
    c, g = _config(case), _generator(seed)
    h, hd, ff = c["hidden_size"], c["head_dim"], c["intermediate_size"]
    qk, kv = c["num_heads"] * hd, c["num_kv_heads"] * hd
    n = case["context"] + case["rows"]

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    w = {name: (rows, k, _pack(c["quant"], 0.02 * normal(rows, k)))
         for name, rows, k in (("q", qk, h), ("k", kv, h), ("v", kv, h), ("o", h, qk), ("gate", ff, h), ("up", ff, h), ("down", h, ff))}
    t = {"x": normal(case["rows"], h), "norm1": 1 + 0.1 * normal(h), "norm2": 1 + 0.1 * normal(h), "kc": normal(n, kv).to(torch.float16), "vc": normal(n, kv).to(torch.float16)}
    return c, w, t


# --------------------------------------------------------------------------------------------------------------------------- run
class _Held:
    """A program's handles, released with it."""

    def __init__(self, **k):
        self.__dict__.update(k)

    def __del__(self):
        for p in getattr(self, "packed", {}).values():
            lib.forge_packed_destroy(p)
        for n in ("engine", "cache", "model"):
            if getattr(self, n, None) is not None:
                getattr(self, n).close()


def prepare(case, seed):
    torch.cuda.empty_cache()
    if case["path"] == "layer":
        c, w, t = _layer_inputs(case, seed)
        packed = {}
        for name, (rows, k, raw) in w.items():
            packed[name] = C.c_void_p()
            check(lib.forge_packed_create(c["quant"], raw.data_ptr(), k, rows, None, C.byref(packed[name])))
        table = np.empty((case["context"] + case["rows"], c["head_dim"] // 2, 2), np.float32)
        check(lib.forge_rope_table(table.ctypes.data, table.shape[0], c["head_dim"], c["rope_theta"]))
        t["table"] = torch.from_numpy(table).cuda()
        m, kv = case["rows"], c["num_kv_heads"] * c["head_dim"]
        for name, n in (("hidden", c["hidden_size"]), ("normed", c["hidden_size"]), ("part", c["hidden_size"]), ("q", c["num_heads"] * c["head_dim"]), ("k", kv), ("v", kv),
                        ("attn", c["num_heads"] * c["head_dim"]), ("gate", c["intermediate_size"]), ("up", c["intermediate_size"]), ("act", c["intermediate_size"])):
            t[name] = torch.empty(m, n, device="cuda")
        return _Held(path="layer", c=c, t=t, packed=packed, rows=m, context=case["context"])
    if case["path"] == "request":
        c = _config(case)
        model = Model(c, _image(c, seed))
        prompts = _prompts(case, c["vocab_size"], seed)
        cache = model.new_cache(max_seq=case["longest"] + case["new"] + 8, batch=case["batch"])
        return _Held(path="request", model=model, cache=cache, prompts=prompts, new=case["new"])
    cfg = _stack_config(case)
    folder = tempfile.mkdtemp(prefix="stack_")
    try:
        _write_folder(folder, cfg, _stack_tensors(cfg, seed))
        model = Model.open(folder, "bfloat16")
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    prompts, follow = _prompts(case, 32768, seed), _follow_ups(case, 32768, seed)
    if case["batch"] == 1:
        return _Held(path="forward", model=model, cache=model.new_cache(max_seq=case["longest"] + case["new"] + 8), prompts=prompts, follow=follow[0].tolist())
    pages = sum(-(-(len(p) + case["new"]) // 64) for p in prompts)
    return _Held(path="steps", model=model, engine=Engine(model, 64 * pages, case["batch"]), plan=_plan(case, prompts, follow), batch=case["batch"])


def _run_layer(s):
    c, t, w, m, base = s.c, s.t, s.packed, s.rows, s.context
    h, hd, nq, nkv, ff = c["hidden_size"], c["head_dim"], c["num_heads"], c["num_kv_heads"], c["intermediate_size"]
    st = torch.cuda.current_stream().cuda_stream
    p = {k: v.data_ptr() for k, v in t.items()}

    def product(out, x, name):
        check(lib.forge_matmul_mat_packed(p[out], m, p[x], w[name], st))

    t["hidden"].copy_(t["x"])
    check(lib.forge_rms_norm(p["normed"], p["hidden"], p["norm1"], m, h, c["rms_norm_eps"], st))
    for name in "qkv":
        product(name, "normed", name)
    check(lib.forge_rope(p["q"], m, base, hd, nq, p["table"], st))
    check(lib.forge_rope(p["k"], m, base, hd, nkv, p["table"], st))
    check(lib.forge_kv_append_f16(p["kc"], p["vc"], p["k"], p["v"], m, base, nkv * hd, st))
    if m == 1:
        check(lib.forge_attention_flash(p["attn"], p["q"], p["kc"], p["vc"], base + 1, nq, nkv, hd, st))
    else:
        check(lib.forge_attention_flash_batch(p["attn"], p["q"], p["kc"], p["vc"], m, base, nq, nkv, hd, st))
    product("part", "attn", "o")
    check(lib.forge_residual_add(p["hidden"], p["part"], m * h, st))
    check(lib.forge_rms_norm(p["normed"], p["hidden"], p["norm2"], m, h, c["rms_norm_eps"], st))
    product("gate", "normed", "gate")
    product("up", "normed", "up")
    check(lib.forge_silu_mul(p["act"], p["gate"], p["up"], m * ff, st))
    product("part", "act", "down")
    check(lib.forge_residual_add(p["hidden"], p["part"], m * h, st))
    return {"hidden": t["hidden"], "k": t["kc"], "v": t["vc"]}


def _run_request(s):
    s.cache.reset()
    if not s.new:
        return {"logits": np.stack([s.model.forward_prefill(p, s.cache, seq=i) for i, p in enumerate(s.prompts)])}
    if len(s.prompts) == 1:
        tokens = s.model.generate_greedy(s.prompts[0], s.new, s.cache)[:, None]
    else:
        first = [int(s.model.forward_prefill(p, s.cache, seq=i).argmax()) for i, p in enumerate(s.prompts)]
        tokens = s.model.decode_greedy_batch(first, s.new, s.cache)
    nxt = [p[0] for p in s.prompts]   # the next turn begins: the caller appends a token of its own
    return {"tokens": tokens.astype(np.int64), "logits": s.model.forward_batch(nxt, s.cache)}


def _run_forward(s):
    s.cache.reset()
    rows = [s.model.forward_prefill(s.prompts[0], s.cache)]
    rows += [s.model.forward(t, s.cache) for t in s.follow]
    return {"logits": np.stack(rows)}


def _run_steps(s):
    got = [[] for _ in range(s.batch)]
    for step in s.plan:
        for (r, _, _), rows in zip(step, s.engine.step(step)):
            if len(rows):
                got[r].append(rows[-1])
    for r in range(s.batch):
        s.engine.release(r)
    return {"logits": np.stack([np.stack(g) for g in got])}


def run(state):
    return {"layer": _run_layer, "request": _run_request, "forward": _run_forward, "steps": _run_steps}[state.path](state)


# ------------------------------------------------------------------------------------------------------------- work and tolerance
def _stack_matrix_values(cfg):
    """Values of the matrices that a token meets (used experts counted once), over all layer runs."""
    shapes = synth.stack_shapes(cfg)
    loop = cfg.get("loop")
    total = shapes["head"][0] * shapes["head"][1]
    for i, L in enumerate(cfg["layers"]):
        times = loop["times"] if loop and loop["start"] <= i < loop["stop"] else 1
        moe = (L.get("mlp") or {}).get("kind") == "moe"
        share = L["mlp"]["router"]["top"] / L["mlp"]["router"]["experts"] if moe else 1.0
        for n, s in shapes.items():
            if n.startswith(f"l{i}.") and len(s) >= 2:
                total += times * s[0] * s[1] * (share if ".mlp.e" in n else 1.0)
    return total


def work(case):
    """Every weight once per pass over it (the prompt of a sequence, or a decoded token of all sequences), cached keys and values once per token that
    reads them; two operations per weight and row, four per query, key and value."""
    if case["path"] == "stack":
        cfg, lens = _stack_config(case), _lengths(case)
        vals = _stack_matrix_values(cfg)
        head = 32768 * case["width"]
        rows = sum(lens) + case["batch"] * case["new"]
        wide = case["heads"] * 2 * 128 * (cfg["layers"][0]["mixer"]["heads"] / case["heads"])
        pairs = sum((n + case["new"]) ** 2 / 2 for n in lens)
        passes = case["new"] + -(-sum(lens) // case["budget"])
        return {"bytes": 2.0 * vals * passes, "flops": 2.0 * (vals - head) * rows + 2.0 * head * case["batch"] * (case["new"] + 1) + case["layers"] * 2.0 * wide * pairs}
    c = _config(case)
    h, qk, kv, ff = c["hidden_size"], c["num_heads"] * c["head_dim"], c["num_kv_heads"] * c["head_dim"], c["intermediate_size"]
    per = h * qk + 2 * h * kv + qk * h + 3 * h * ff
    if case["path"] == "layer":
        m, n = case["rows"], case["rows"] + case["context"]
        return {"bytes": per * configs.block_bytes(c) / 32 + 8.0 * m * h + 4.0 * kv * n, "flops": 2.0 * m * per + 4.0 * qk * m * (n - (m - 1) / 2)}
    pq = configs.proj_quants(c)
    row = lambda cat, k: configs.raw_row_bytes(pq[cat], k)  # noqa: E731
    layer = qk * row(0, h) + kv * (row(1, h) + row(2, h)) + h * row(3, qk) + ff * (row(4, h) + row(5, h)) + h * row(6, ff)
    weights = layer * c["num_layers"] + c["vocab_size"] * row(7, h)
    steps = case["new"] + 1 if case["new"] else 0
    nbytes = flops = 0.0
    for n in _lengths(case):
        nbytes += weights
        flops += configs.prefill_flops(c, n) + steps * 2.0 * (per * c["num_layers"] + h * c["vocab_size"])
        nbytes += c["num_layers"] * 4.0 * kv * sum(n + i for i in range(steps))
    return {"bytes": nbytes + weights * steps, "flops": flops}


def tolerance(case):
    """About four times what the paths are off a 64-bit computation: 2e-4 for a layer (the cache is fp16), 5e-4 for quantised models, 3e-3 and
    1e-2 for the bfloat16 ones (where two experts' scores are close, rounding decides).  Rows of K-quant products are rounded to 8 bits,
    and a last bit in front of a rounding moves the logits by up to 2.5e-2."""
    if case["path"] == "layer":
        return {"rel": 1e-3}
    if case["path"] == "request":
        return {"rel": 0.03, "max": 0.9, "differ": 0.005} if case["quant"] == "q4_k_m" else {"rel": 2e-3, "differ": 0.005}
    return {"rel": 0.01, "max": 0.4} if case["design"] == "bolenex" else {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------------------------------- exact
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, pos, freq, factor=1.0, pairs=False):
    """Rotates [..., tokens, heads, n]: entries (i, i + n/2), or (2 i, 2 i + 1) with ``pairs``."""
    ang = pos.double()[:, None, None] * freq
    c, s = torch.cos(ang) * factor, torch.sin(ang) * factor
    a, b = (x[..., 0::2], x[..., 1::2]) if pairs else x.chunk(2, -1)
    u, v = a * c - b * s, b * c + a * s
    return torch.stack([u, v], -1).flatten(-2) if pairs else torch.cat([u, v], -1)


def _attend(q, k, v, scale, first=0, size=None, keep=0, sink=None):
    """q: [tokens, heads, d]; query i stands at position first + i."""
    n, H, _ = q.shape
    rep = H // k.shape[1]
    i, j = torch.arange(n, device="cuda")[:, None] + first, torch.arange(k.shape[0], device="cuda")[None]
    see = j <= i
    if size is not None:
        see &= (i - j < size) | (j < keep)
    out = []
    for hd in range(H):
        s = (q[:, hd] @ k[:, hd // rep].T * scale).masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[hd].expand(n, 1)], 1)
        out.append(torch.softmax(s, 1)[:, :k.shape[0]] @ v[:, hd // rep])
    return torch.stack(out, 1)


def _decoder_rows(c, t, tokens):
    """Final normed rows of the tokens of one sequence."""
    eps, hd, nq, nkv = c["rms_norm_eps"], c["head_dim"], c["num_heads"], c["num_kv_heads"]
    pos = torch.arange(len(tokens), device="cuda")
    freq = c["rope_theta"] ** (-2.0 * torch.arange(hd // 2, device="cuda", dtype=torch.float64) / hd)
    pq = configs.proj_quants(c)

    def product(x, name, cat):
        if pq[cat] in (Q4_K, Q6_K):   # these products are defined on rows rounded to blocks of 32 int8 values
            b = x.float().reshape(-1, 32)
            d, inv = _scales_q8(b)
            x = (torch.clamp(torch.round(b * inv[:, None]), -127, 127).double() * d.half().double()[:, None]).reshape(x.shape)
        return x @ t[name].T

    x = t["embed"][tokens].double()
    for i in range(c["num_layers"]):
        y = _rms(x, t[f"{i}.attn_norm"], eps)
        q, k, v = (product(y, f"{i}.{n}", cat) + (t[f"{i}.{n}b"] if c["qkv_bias"] else 0) for cat, n in enumerate("qkv"))
        q, k = (_turn(a.reshape(-1, heads, hd), pos, freq, pairs=True) for a, heads in ((q, nq), (k, nkv)))
        x = x + product(_attend(q, k, v.reshape(-1, nkv, hd), hd ** -0.5).flatten(1), f"{i}.o", 3)
        y = _rms(x, t[f"{i}.ffn_norm"], eps)
        g = product(y, f"{i}.gate", 4)
        x = x + product(g * torch.sigmoid(g) * product(y, f"{i}.up", 5), f"{i}.down", 6)
    y = _rms(x, t["norm"], eps)
    return y, lambda rows: product(rows, "head", 7)


def _exact_request(case, seed):
    c = _config(case)
    t = {n: (_unpack(quant, x, rows) if quant else x if n == "embed" else x.double()) for n, quant, rows, x in _decoder_tensors(c, seed)}
    nxt = _successors(seed, c["vocab_size"]).cpu().numpy()
    tokens, logits = [], []
    for p in _prompts(case, c["vocab_size"], seed):
        chain = [int(p[-1])]
        for _ in range(case["new"]):
            chain.append(int(nxt[chain[-1]]))
        seq = np.concatenate([p, np.array(chain[1:], np.uint32), p[:1]]) if case["new"] else p
        rows, head = _decoder_rows(c, t, torch.from_numpy(seq.astype(np.int64)).cuda())
        if not case["new"]:
            logits.append(head(rows[-1:])[0].cpu().numpy())
            continue
        z = head(rows[len(p) - 1:])
        if z[:-2].argmax(1).cpu().tolist() != chain[1:]:
            raise RuntimeError("a token does not follow from its predecessor: the chain is not the greedy one")
        tokens.append(chain[1:])
        logits.append(z[-1].cpu().numpy())
    return {"tokens": np.array(tokens, np.int64).T, "logits": np.stack(logits)} if case["new"] else {"logits": np.stack(logits)}


def _exact_layer(case, seed):
    c, w, t = _layer_inputs(case, seed)
    hd, nq, nkv, eps, base = c["head_dim"], c["num_heads"], c["num_kv_heads"], c["rms_norm_eps"], case["context"]
    w = {n: _unpack(c["quant"], raw, rows) for n, (rows, _, raw) in w.items()}
    t = {n: x.double() for n, x in t.items()}
    pos = torch.arange(base, base + case["rows"], device="cuda")
    freq = c["rope_theta"] ** (-2.0 * torch.arange(hd // 2, device="cuda", dtype=torch.float64) / hd)
    y = _rms(t["x"], t["norm1"], eps)
    q, k = (_turn((y @ w[a].T).reshape(-1, heads, hd), pos, freq, pairs=True) for a, heads in (("q", nq), ("k", nkv)))
    kc, vc = t["kc"], t["vc"]
    kc[base:], vc[base:] = k.flatten(1), y @ w["v"].T
    o = _attend(q, kc.reshape(-1, nkv, hd), vc.reshape(-1, nkv, hd), hd ** -0.5, base)
    x = t["x"] + o.flatten(1) @ w["o"].T
    y = _rms(x, t["norm2"], eps)
    g = y @ w["gate"].T
    return {"hidden": x + (g * torch.sigmoid(g) * (y @ w["up"].T)) @ w["down"].T, "k": kc, "v": vc}


def _latent_mixer(h, w, m, eps):
    n, H, d, r, rank = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    pos = torch.arange(n, device="cuda")
    freq = m["rot"]["base"] ** (-2.0 * torch.arange(r // 2, device="cuda", dtype=torch.float64) / r)
    q, down = (h @ w("q").T).reshape(n, H, d + r), h @ w("dkv").T
    c = _rms(down[:, :rank], w("dkv.norm"), eps)
    kr = _turn(down[:, None, rank:], pos, freq).expand(n, H, r)
    q = torch.cat([q[..., :d], _turn(q[..., d:], pos, freq)], -1)
    k = torch.cat([(c @ w("uk").T).reshape(n, H, d), kr], -1)
    o = _attend(q, k, (c @ w("uv").T).reshape(n, H, m["vdim"]), m["scale"]).flatten(1)
    return (o * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _softmax_mixer(h, w, L, eps):
    m, n = L["mixer"], h.shape[0]
    H, G, d, s = m["heads"], m["kv_heads"], m["dim"], m["rot"]["scaling"]
    pos, i = torch.arange(n, device="cuda"), torch.arange(d // 2, device="cuda", dtype=torch.float64)
    freq = m["rot"]["base"] ** (-2.0 * i / d)
    if L["type"] == "attention":     # norms per head, interleaved pairs, YaRN frequencies, a window with kept tokens and a learned sink
        turns = lambda x: d * math.log(s["original"] / (2 * math.pi * x)) / (2 * math.log(m["rot"]["base"]))  # noqa: E731
        lo, hi = max(math.floor(turns(s["fast"])), 0), min(math.ceil(turns(s["slow"])), d - 1)
        ramp = torch.clamp((i - lo) / max(hi - lo, 0.001), 0, 1)
        freq, factor = freq / s["factor"] * ramp + freq * (1 - ramp), 0.1 * math.log(s["factor"]) + 1
        q, k = ((h @ w(x).T).reshape(n, g, d) for x, g in (("q", H), ("k", G)))
        q, k = (_turn(_rms(x, w(y), eps), pos, freq, factor, True) for x, y in ((q, "q.norm"), (k, "k.norm")))
        o = _attend(q, k, (h @ w("v").T).reshape(n, G, -1), m["scale"], 0, m["mask"]["size"], m["mask"]["keep_first"], w("sink"))
    else:                            # norms over all heads, biases, rotated halves, linear scaling, a sink of score zero
        q, k, v = (h @ w(x).T + w(x + ".b") for x in "qkv")
        q, k = (_turn(_rms(x, w(y), eps).reshape(n, g, d), pos, freq / s["factor"]) for x, y, g in ((q, "q.norm", H), (k, "k.norm", G)))
        o = _attend(q, k, v.reshape(n, G, -1), m["scale"], sink=torch.zeros(H, device="cuda", dtype=torch.float64))
    return o.flatten(1) @ w("o").T


def _linear_mixer(hs, w, m, eps):
    """Gated linear attention of several sequences side by side (their ends padded)."""
    n, B, H, d, dv = max(len(h) for h in hs), len(hs), m["heads"], m["dim"], m["vdim"]
    h = torch.nn.utils.rnn.pad_sequence(hs, batch_first=True)
    q, k, v = ((h @ w(x).T).reshape(B, n, H, -1) for x in "qkv")
    a = torch.sigmoid(((h @ w("a1").T) @ w("a2").T + w("a2.b")).reshape(B, n, H, d)) ** (1.0 / m["tau"])
    S = torch.zeros(B, H, d, dv, device="cuda", dtype=torch.float64)
    o = torch.empty(B, n, H, dv, device="cuda", dtype=torch.float64)
    for t in range(n):
        S = torch.baddbmm((a[:, t, :, :, None] * S).flatten(0, 1), k[:, t].reshape(B * H, d, 1), v[:, t].reshape(B * H, 1, dv)).reshape(B, H, d, dv)
        o[:, t] = (q[:, t].reshape(B * H, 1, d) @ S.flatten(0, 1)).reshape(B, H, dv) * d ** -0.5
    gate = h @ w("g").T
    o = (_rms(o, w("norm"), eps).flatten(2) * gate * torch.sigmoid(gate)) @ w("o").T
    return [o[b, :len(x)] for b, x in enumerate(hs)]


def _silu_glu(h, w):
    g = h @ w("gate").T
    return (g * torch.sigmoid(g) * (h @ w("up").T)) @ w("down").T


def _experts(h, w, m):
    z = h @ w("router").T + w("router.b")
    val, idx = z.topk(m["router"]["top"], 1)
    val = torch.softmax(val, 1)
    out = torch.zeros_like(h)
    for e in range(z.shape[1]):
        at, which = (idx == e).nonzero(as_tuple=True)
        if len(at):
            out.index_add_(0, at, val[at, which][:, None] * _silu_glu(h[at], lambda n: w(f"e{e}.{n}")))
    return out


def _exact_stack(case, seed):
    cfg = _stack_config(case)
    t = {n: x.double() for n, x in _stack_tensors(cfg, seed).items()}
    prompts, follow, eps = _prompts(case, 32768, seed), _follow_ups(case, 32768, seed), cfg["norm"]["eps"]
    seqs = [torch.from_numpy(np.concatenate([p, f]).astype(np.int64)).cuda() for p, f in zip(prompts, follow)]
    mokatar = cfg["architecture"] == "Mokatar"
    xs = [t["embed"][s] for s in seqs]
    if mokatar:
        b = cfg["embedding"]["bigram"]
        rows = [torch.cat([s.new_full((1,), b["buckets"]), (s[:-1] * b["mul_prev"] + s[1:] * b["mul_cur"]) % b["buckets"]]) for s in seqs]
        xs = [x * cfg["embedding"]["scale"] + t["bigram"][r] for x, r in zip(xs, rows)]
    start = xs

    def norm(x, name):
        if mokatar:
            return _rms(x, 1 + t[name], eps)
        return torch.tanh(t[name + ".alpha"] * x) * t[name] + t[name + ".b"]

    loop = cfg.get("loop")
    order = [(i, None) for i in range(len(cfg["layers"]))]
    if loop:
        body = [(i, n if i == loop["start"] else None) for n in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
        order = order[:loop["start"]] + body + order[loop["stop"]:]
    for i, entry in order:
        L = cfg["layers"][i]
        mix, mlp = (lambda n: t[f"l{i}.mix.{n}"]), (lambda n: t[f"l{i}.mlp.{n}"])
        if entry is not None:
            xs = [(x + x0 if entry else x) + t["loop.step"][entry] for x, x0 in zip(xs, start)]
        hs = [norm(x, f"l{i}.norm1") for x in xs]
        if L["type"] == "gla":
            ys = _linear_mixer(hs, mix, L["mixer"], eps)
        elif mokatar:
            ys = [_softmax_mixer(h, mix, L, eps) for h in hs]
        else:
            ys = [_latent_mixer(h, mix, L["mixer"], eps) for h in hs]
        if mokatar:
            fs = [norm(x, f"l{i}.norm2") for x in xs]
            fs = [_experts(f, mlp, L["mlp"]) if L["mlp"]["kind"] == "moe" else _silu_glu(f, mlp) for f in fs]
        else:
            fs = []
            for h in hs:
                g, u = torch.clamp(h @ mlp("gate").T, max=L["mlp"]["limit"]), torch.clamp(h @ mlp("up").T, -L["mlp"]["limit"], L["mlp"]["limit"])
                fs.append((g * torch.sigmoid(1.702 * g) * (u + 1)) @ mlp("down").T)
        xs = [x + y + f for x, y, f in zip(xs, ys, fs)]
    scale = cfg.get("logit_scale", 1.0)
    return {"logits": np.stack([(norm(x[len(p) - 1:], "final.norm") @ t["head"].T * scale).cpu().numpy() for x, p in zip(xs, prompts)])}


def exact(case, seed):
    torch.cuda.empty_cache()
    return {"request": _exact_request, "layer": _exact_layer, "stack": _exact_stack}[case["path"]](case, seed)
