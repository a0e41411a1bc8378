"""The work that users of this package have it do, as timed and compared cases.

Four families, each through the public entry points:

  chain   the block mat-vecs of decode steps: prepared descriptors over as many distinct weights as keep them out of L2, recorded
          into one CUDA graph (ops.make_desc, ops.launch); 1 to 64 activation rows
  gemm    the projections of a prompt, one eager ops.qmatmul per weight
  llama   LlamaDecoder over Q8_0 / Q4_0 / Q4_K blocks: a prompt as one batch, or recorded decode steps fed given tokens
  layers  LayerListDecoder (Bigerax: windows and gated recurrences; Lenesun: latent attention and mixtures of experts): a prompt,
          or a reply (a prompt, then given tokens one at a time)

Tokens fall into clusters and each router knows them, as trained ones do: its choices are clear and the experts evenly used.
Weights are drawn with zero mean and a spread of K^-1/2, as trained matrices have them, so that activations keep their size from
layer to layer.  Tokens of decode steps are given rather than picked, so that two correct implementations see the same input.
`exact` is the same arithmetic in 64 bits, from the formats' and models' definitions alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cut_b200 import _lib as L
from cut_b200 import ops
from cut_b200.layer_list import (Bigram, FeedForward, GatedRecurrence, LatentAttention, Layer, LayerListConfig, LayerListDecoder,
                                 MixtureOfExperts, Rotation, WindowAttention)
from cut_b200.llama_decode import LlamaConfig, LlamaDecoder

FORMATS = {"Q8_0": (L.Q8_0, 32, 34), "Q4_0": (L.Q4_0, 32, 18), "Q4_K": (L.Q4_K, 256, 144)}  # code, weights and bytes per block
SILU, ADD = 133, 0  # operator codes of the fused epilogues


def listed():
    llama = {"kind": "llama", "hidden": 4096, "heads": 32, "kv_heads": 8, "head": 128, "ffn": 14336, "vocab": 32000}
    return [
        # one decode step's projections over an 8-bit 4096 x 4096 model, fp32 activations: the smallest launches
        {"name": "q8_matvec_4096", "kind": "chain", "fmt": "Q8_0", "rows": 1, "K": 4096, "N": 4096, "act": "f32", "count": 16, "fuse": "none"},
        # a 7B model's feed-forward projections at batch 1
        {"name": "q4_matvec_11008", "kind": "chain", "fmt": "Q4_0", "rows": 1, "K": 4096, "N": 11008, "act": "f16", "count": 32, "fuse": "none"},
        # a 70B model's gate / up projections at batch 1
        {"name": "q4_matvec_28672", "kind": "chain", "fmt": "Q4_0", "rows": 1, "K": 8192, "N": 28672, "act": "f16", "count": 8, "fuse": "none"},
        # eight sequences decoded together
        {"name": "q4_batch8_11008", "kind": "chain", "fmt": "Q4_0", "rows": 8, "K": 4096, "N": 11008, "act": "f16", "count": 32, "fuse": "none"},
        # thirty-two sequences decoded together, a 70B model's square projections
        {"name": "q4_batch32_8192", "kind": "chain", "fmt": "Q4_0", "rows": 32, "K": 8192, "N": 8192, "act": "f16", "count": 16, "fuse": "none"},
        # the feed-forward projection of a 512-token prompt
        {"name": "q4k_gemm_512", "kind": "gemm", "fmt": "Q4_K", "rows": 512, "K": 4096, "N": 14336, "act": "f16", "count": 4, "fuse": "none"},
        # a ragged prompt through an 8-bit down projection with the residual add fused, fp32 activations
        {"name": "q8_gemm_333_add", "kind": "gemm", "fmt": "Q8_0", "rows": 333, "K": 11008, "N": 4096, "act": "f32", "count": 4, "fuse": "add"},
        # eight layers of an 8B-sized decoder: a 512-token prompt, and tokens after it
        {**llama, "name": "llama_prefill_512", "fmt": "Q4_K", "layers": 8, "prompt": 512, "steps": 0},
        {**llama, "name": "llama_decode", "fmt": "Q4_K", "layers": 8, "prompt": 512, "steps": 16},
        # a long prompt through windows and recurrences
        {"name": "bigerax_prefill_2048", "kind": "layers", "model": "bigerax", "dtype": "bfloat16", "width": 4096, "heads": 32, "kv_heads": 8,
         "head": 128, "ffn": 14336, "window": 1024, "layers": 16, "vocab": 32000, "prompt": 2048, "want": 1, "steps": 0},
        # a long prompt of an odd length through latent attention and experts, its last places scored
        {"name": "lenesun_prefill_1501", "kind": "layers", "model": "lenesun", "dtype": "bfloat16", "width": 4096, "heads": 32, "head": 128,
         "rot": 64, "q_rank": 1536, "rank": 512, "experts": 16, "top": 4, "ffn": 2048, "layers": 8, "vocab": 32000, "prompt": 1501, "want": 32,
         "steps": 0},
        # a short prompt and the reply to it
        {"name": "lenesun_reply", "kind": "layers", "model": "lenesun", "dtype": "bfloat16", "width": 4096, "heads": 32, "head": 128,
         "rot": 64, "q_rank": 1536, "rank": 512, "experts": 16, "top": 4, "ffn": 2048, "layers": 8, "vocab": 32000, "prompt": 200, "want": 1,
         "steps": 24},
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step) * step))


def draw(rng):
    kind = rng.choice(["chain", "chain", "chain", "gemm", "gemm", "gemm", "llama", "llama", "layers", "layers", "layers"])
    if kind in ("chain", "gemm"):
        fmt = rng.choice(["Q8_0", "Q4_0", "Q4_K"])
        ragged = fmt != "Q4_K" and rng.random() < 0.25  # widths of whole 32-weight blocks and no more, as some small models have
        K = _log_int(rng, 512, 4096, 32) if ragged else _log_int(rng, 1024, 14336, 256)
        N = _log_int(rng, 1000, 4096 if ragged else 28672, rng.choice([1, 16, 256]))
        case = {"kind": kind, "fmt": fmt, "K": K, "N": N, "act": rng.choice(["f16", "f32"]), "fuse": rng.choice(["none", "none", "silu", "add"])}
        if kind == "chain":
            size = N * K // FORMATS[fmt][1] * FORMATS[fmt][2]
            return {**case, "rows": rng.choice([1, 1, 2, 3, 4, 8, rng.randint(5, 16), _log_int(rng, 17, 64)]), "count": max(2, min(32, int(500e6 // size)))}
        return {**case, "rows": _log_int(rng, 17, 384 if ragged else 2048), "count": 1 if ragged else 3}
    if kind == "llama":
        heads, kv_heads, head = rng.choice([(32, 8, 128), (16, 4, 128), (16, 16, 128), (16, 2, 64), (24, 8, 128)])
        hidden = heads * head
        prompt = _log_int(rng, 17, 1500)
        return {"kind": "llama", "hidden": hidden, "heads": heads, "kv_heads": kv_heads, "head": head, "ffn": _log_int(rng, 2048, 11008, 256),
                "vocab": rng.randint(4000, 32000), "fmt": rng.choice(["Q8_0", "Q4_0", "Q4_K"]), "layers": rng.randint(2, 4), "prompt": prompt,
                "steps": rng.choice([0, rng.randint(4, 12)])}
    narrow = rng.random() < 0.25  # the 32-bit mode, on small models
    case = {"kind": "layers", "model": rng.choice(["bigerax", "lenesun"]), "dtype": "float32" if narrow else "bfloat16",
            "width": rng.choice([1024] if narrow else [1024, 2048, 2560, 4096]), "layers": rng.randint(2, 4), "vocab": rng.randint(4000, 32000),
            "prompt": _log_int(rng, 16, 200 if narrow else 2048), "want": rng.choice([1, 8])}
    case["steps"] = rng.choice([0, rng.randint(4, 16)])
    case["want"] = min(case["want"], case["prompt"])
    if case["model"] == "bigerax":
        heads, kv_heads, head = rng.choice([(8, 2, 128), (16, 4, 128), (32, 8, 128), (16, 8, 64), (12, 4, 96)])
        return {**case, "heads": heads, "kv_heads": kv_heads, "head": head, "window": _log_int(rng, 64, 2048), "ffn": _log_int(rng, 2048, 8192, 8)}
    return {**case, "heads": rng.choice([8, 16, 32]), "head": rng.choice([64, 128]), "rot": rng.choice([32, 64]),
            "q_rank": rng.choice([512, 768, 1536]), "rank": rng.choice([256, 512]), "experts": rng.choice([8, 16, 32]), "top": rng.choice([2, 4]),
            "ffn": _log_int(rng, 512, 2048, 8)}


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *shape, scale=1.0):
    return torch.randn(shape, device="cuda", generator=g).mul_(scale)


def _bytes(g, lo, hi, *shape):
    return torch.randint(lo, hi, shape, dtype=torch.int16, device="cuda", generator=g)


def _blocks(g, fmt, N, K):
    """N rows of K weights as blocks (flat bytes): uniform quants, scales around what gives the weights a spread of K^-1/2."""
    _, per, size = FORMATS[fmt]
    nb = N * K // per
    out = torch.empty((nb, size), dtype=torch.uint8, device="cuda")
    half = lambda x: x.to(torch.float16).view(torch.uint8).reshape(nb, 2)
    spread = torch.rand(nb, device="cuda", generator=g).mul_(0.5).add_(0.75) * K ** -0.5
    if fmt == "Q8_0":
        out[:, :2] = half(spread / 73.6)
        out[:, 2:] = _bytes(g, -127, 128, nb, 32).to(torch.int8).view(torch.uint8)
    elif fmt == "Q4_0":
        out[:, :2] = half(spread / 4.3)
        out[:, 2:] = (_bytes(g, 1, 16, nb, 16) | (_bytes(g, 1, 16, nb, 16) << 4)).to(torch.uint8)  # -7 .. 7
    else:  # sub-blocks with scales 32 .. 63 and minima 7.5 d sc, the middle of the quants
        d = spread / (4.6 * 47.5)
        out[:, :2], out[:, 2:4] = half(d), half(7.5 * d)
        sc = _bytes(g, 32, 64, nb, 8)
        for at in (0, 4):  # scales, then minima: both are sc
            out[:, 4 + at: 8 + at] = (sc[:, :4] | (sc[:, 4:] >> 4 << 6)).to(torch.uint8)
        out[:, 12:16] = ((sc[:, 4:] & 15) | ((sc[:, 4:] & 15) << 4)).to(torch.uint8)
        out[:, 16:] = _bytes(g, 0, 256, nb, 128).to(torch.uint8)
    return out.reshape(-1)


def _matmul_inputs(case, seed):
    g = _gen(seed)
    N, K, rows = case["N"], case["K"], case["rows"]
    act = torch.float16 if case["act"] == "f16" else torch.float32
    W = [_blocks(g, case["fmt"], N, K) for _ in range(case["count"])]
    A = [_rand(g, rows, K).to(act) for _ in range(case["count"])]
    D = [_rand(g, rows, N) for _ in range(case["count"])] if case["fuse"] == "add" else [None] * case["count"]
    return W, A, D


def _fusion(case):
    return {"none": {}, "silu": {"fusion_type": L.FUSION_UNARY, "fusion_op": SILU}, "add": {"fusion_type": L.FUSION_BINARY, "fusion_op": ADD}}[case["fuse"]]


def _llama_config(case):
    return LlamaConfig(n_layers=case["layers"], hidden=case["hidden"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], head_dim=case["head"],
                       ffn=case["ffn"], vocab=case["vocab"], max_seq=case["prompt"] + case["steps"] + 8, fmt=FORMATS[case["fmt"]][0])


def _llama_shapes(case):
    q, kv = case["heads"] * case["head"], case["kv_heads"] * case["head"]
    return {"wqkv": (q + 2 * kv, case["hidden"]), "wo": (case["hidden"], q), "wgate": (case["ffn"], case["hidden"]),
            "wup": (case["ffn"], case["hidden"]), "wdown": (case["hidden"], case["ffn"])}


def _llama_inputs(case, seed):
    """Weights on the device, and the tokens."""
    g = _gen(seed)
    norm = lambda: 1.0 + 0.1 * _rand(g, case["hidden"])
    layers = [{**{k: _blocks(g, case["fmt"], *s) for k, s in _llama_shapes(case).items()}, "attn_norm": norm(), "ffn_norm": norm()}
              for _ in range(case["layers"])]
    w = {"layers": layers, "final_norm": norm(), "lm_head": _blocks(g, case["fmt"], case["vocab"], case["hidden"]),
         "embedding": _rand(g, case["vocab"], case["hidden"])}
    tokens = np.random.default_rng(seed).integers(0, case["vocab"], case["prompt"] + max(case["steps"], 1))
    return w, tokens


def _layer_config(case):
    W, n = case["width"], case["layers"]
    if case["model"] == "bigerax":
        att = WindowAttention(case["heads"], case["kv_heads"], case["head"], case["head"], case["window"], case["head"] ** -0.5,
                              Rotation(10000.0, case["head"]), True, True)
        layers = [Layer(GatedRecurrence(W), None) if i % 4 == 0 else Layer(att, FeedForward(case["ffn"])) for i in range(n)]
        return LayerListConfig(W, case["vocab"], tuple(layers), 2, 1e-6, Bigram(65521, 36313, 27191))
    wide = case["head"] + case["rot"]
    att = lambda j: LatentAttention(case["heads"], case["head"], case["head"], case["q_rank"], case["rank"], wide ** -0.5,
                                    Rotation(10000.0, case["rot"]), True, j)
    moe = MixtureOfExperts(case["experts"], case["top"], case["ffn"], 7.0, 1.702, 1.0)
    layers = tuple(Layer(att(None if i % 2 == 0 else i - 1), moe) for i in range(n))
    return LayerListConfig(W, case["vocab"], layers, 1, 1e-6, norm_center=True, parallel=True, residual_mult=0.4, embed_scale=2.0, tied_head=True)


def _layer_inputs(case, seed):
    g, cfg = _gen(seed), _layer_config(case)
    mat = lambda *s: _rand(g, *s, scale=s[-1] ** -0.5).to(torch.bfloat16)
    one = lambda n: 1.0 + 0.1 * _rand(g, n)
    W, layers = cfg.width, []
    embed, clusters = _rand(g, cfg.vocab, W), _rand(g, 64, W)
    if any(isinstance(l.mlp, MixtureOfExperts) for l in cfg.layers):
        embed += clusters[torch.arange(cfg.vocab, device="cuda") % 64]
    for l in cfg.layers:
        m, f, d = l.mixer, l.mlp, {"norm1": one(W)}
        if isinstance(m, GatedRecurrence):
            d["mix"] = {"z": mat(m.width, W), "x": mat(m.width, W), "g": mat(m.width, W), "o": mat(W, m.width)}
        elif isinstance(m, WindowAttention):
            d["mix"] = {"q": mat(m.q_rows, W), "k": mat(m.k_rows, W), "v": mat(m.v_rows, W), "o": mat(W, m.heads * m.vdim), "vmix": 0.3}
            d["mix"].update({n + ".b": 0.1 * _rand(g, r) for n, r in (("q", m.q_rows), ("k", m.k_rows), ("v", m.v_rows), ("o", W))})
        else:
            d["mix"] = {"dq": mat(m.q_rank, W), "dq.norm": one(m.q_rank), "uq": mat(m.q_rows, m.q_rank), "uk": mat(m.heads * m.dim, m.kv_rank),
                        "uv": mat(m.heads * m.vdim, m.kv_rank), "o": mat(W, m.heads * m.vdim), "sink": _rand(g, m.heads)}
            if m.kv_from is None:
                d["mix"].update({"dkv": mat(m.kv_rows, W), "dkv.norm": one(m.kv_rank)})
        if isinstance(f, FeedForward):
            d["mlp"] = {"up": mat(f.ff, W), "down": mat(W, f.ff), "up.b": 0.1 * _rand(g, f.ff), "down.b": 0.1 * _rand(g, W)}
        elif f is not None:
            likes = torch.zeros((64, f.experts), device="cuda").scatter_(1, torch.rand((64, f.experts), device="cuda", generator=g).topk(f.top).indices, 0.25)
            d["mlp"] = {"gate": mat(f.experts, f.ff, W), "up": mat(f.experts, f.ff, W), "down": mat(f.experts, W, f.ff),
                        "router": (likes.T @ clusters).mul_(W ** -0.5).to(torch.bfloat16), "router.b": 0.1 * _rand(g, f.experts)}
        if not cfg.parallel:
            d.update({"norm1b": one(W)}, **({"norm2": one(W), "norm2b": one(W)} if f is not None else {}))
        layers.append(d)
    w = {"embed": embed.to(torch.bfloat16), "final_norm": one(W), "layers": layers}
    if cfg.bigram:
        w.update({"bigram": _rand(g, cfg.bigram.buckets + 1, W).to(torch.bfloat16), "head": mat(cfg.vocab, W)})
    tokens = np.random.default_rng(seed).integers(0, cfg.vocab, case["prompt"] + case["steps"])
    return cfg, w, [int(t) for t in tokens]


def prepare(case, seed):
    if case["kind"] in ("chain", "gemm"):
        W, A, D = _matmul_inputs(case, seed)
        s = {"case": case, "W": W, "A": A, "D": D}
        if case["kind"] == "chain":
            s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
            s["plans"], s["keep"], s["out"] = [], [], []
            for w, a, dd in zip(W, A, D):
                d, out, keep = ops.make_desc(a, w, FORMATS[case["fmt"]][0], case["N"], D=dd, status=s["status"], **_fusion(case))
                need = ops.workspace_bytes(d)
                if need:
                    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
                    d.workspace, d.workspace_bytes = ws.data_ptr(), need
                    keep = keep + (ws,)
                s["plans"].append(d)
                s["keep"].append(keep)
                s["out"].append(out)
            for d in s["plans"]:
                ops.launch(d)
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                for d in s["plans"]:
                    ops.launch(d)
        return s
    if case["kind"] == "llama":
        w, tokens = _llama_inputs(case, seed)
        host = lambda v: {k: host(x) for k, x in v.items()} if isinstance(v, dict) else [host(x) for x in v] if isinstance(v, list) else v.cpu().numpy()
        dec = LlamaDecoder(_llama_config(case), host(w))
        n = case["prompt"]
        s = {"case": case, "dec": dec, "prompt": tokens[:n], "steps": torch.from_numpy(tokens[n:].astype(np.int32)).cuda(), "first": int(tokens[n])}
        if case["steps"]:
            dec.prefill(s["prompt"])
            dec.step(s["first"], n)
            dec.capture()
        return s
    cfg, w, tokens = _layer_inputs(case, seed)
    dec = LayerListDecoder(cfg, w, dtype=case["dtype"], max_seq=len(tokens) + 16)
    s = {"case": case, "dec": dec, "prompt": tokens[: case["prompt"]], "reply": tokens[case["prompt"]:]}
    if case["steps"]:  # a server's first request: the decode step is recorded when it runs a second time
        run({**s, "reply": s["reply"][:2]})
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    if case["kind"] == "chain":
        s["graph"].replay()
        return s["out"]
    if case["kind"] == "gemm":
        fmt, fusion = FORMATS[case["fmt"]][0], _fusion(case)
        return [ops.qmatmul(a, w, fmt, case["N"], D=d, **fusion) for a, w, d in zip(s["A"], s["W"], s["D"])]
    dec = s["dec"]
    if case["kind"] == "llama":
        if case["steps"]:
            dec.set_position(s["first"], case["prompt"])
            for i in range(case["steps"]):
                if i:
                    dec.token.copy_(s["steps"][i: i + 1])
                dec.replay(1)
        else:
            dec.prefill(s["prompt"])
        return {"logits": dec.logits, "k": dec.k_cache, "v": dec.v_cache}
    seq = dec.open()
    n = case["prompt"]
    out = [dec.forward(seq, s["prompt"], range(n - case["want"], n))]
    for t in s["reply"]:
        out.append(dec.forward(seq, [t], [0]).clone())
    dec.close(seq)
    return torch.cat(out)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    if case["kind"] in ("chain", "gemm"):
        _, per, size = FORMATS[case["fmt"]]
        N, K, M = case["N"], case["K"], case["rows"]
        one = N * K // per * size + M * K * (2 if case["act"] == "f16" else 4) + M * N * (8 if case["fuse"] == "add" else 4)
        return {"bytes": case["count"] * one, "flops": 2.0 * case["count"] * M * N * K}
    T, steps = case["prompt"], case["steps"]
    if case["kind"] == "llama":
        _, per, size = FORMATS[case["fmt"]]
        weights = case["layers"] * sum(n * k for n, k in _llama_shapes(case).values())
        head, row = case["vocab"] * case["hidden"], case["kv_heads"] * case["head"] * 4  # row: a position's fp16 keys and values
        pair = 4.0 * case["heads"] * case["head"] * case["layers"]                       # FLOPs of a query and a key
        if steps:
            seen = sum(T + i + 1 for i in range(steps))
            return {"bytes": steps * (weights + head) // per * size + case["layers"] * row * (seen + steps) + steps * 4 * case["vocab"],
                    "flops": 2.0 * steps * (weights + head) + pair * seen}
        return {"bytes": (weights + head) // per * size + 4 * T * case["hidden"] + case["layers"] * row * T + 4 * case["vocab"],
                "flops": 2.0 * (T * weights + head) + pair * T * (T + 1) / 2}
    cfg = _layer_config(case)
    nbytes, flops = 0.0, 0.0
    el = 2 if case["dtype"] == "bfloat16" else 4
    head = cfg.vocab * cfg.width
    for l in cfg.layers:
        m, f = l.mixer, l.mlp
        pairs = lambda n: T * (T + 1) / 2 + sum(T + i + 1 for i in range(n))
        if isinstance(m, GatedRecurrence):
            dense = 4 * m.width * cfg.width
        elif isinstance(m, WindowAttention):
            dense = (m.q_rows + m.k_rows + m.v_rows + m.heads * m.vdim) * cfg.width
            seen = sum(min(m.window, i + 1) for i in range(T + steps))
            flops += 2.0 * m.heads * (m.dim + m.vdim) * seen
            nbytes += m.kv_heads * (m.dim + m.vdim) * el * (T + steps + sum(min(m.window, T + i + 1) for i in range(steps)))
        else:
            dense = (m.q_rank + m.kv_rows + m.heads * m.vdim) * cfg.width + m.q_rows * m.q_rank + m.heads * (m.dim + m.vdim) * m.kv_rank
            flops += 2.0 * m.heads * (m.dim + m.rot.dims + m.vdim) * pairs(steps)
            nbytes += (m.kv_rank + m.rot.dims) * el * (T + sum(T + i + 1 for i in range(steps)))
        if isinstance(f, FeedForward):
            dense += 2 * f.ff * cfg.width
        if isinstance(f, MixtureOfExperts):
            dense += f.experts * cfg.width
            expert = 3 * f.ff * cfg.width
            nbytes += 2.0 * expert * (min(f.experts, T * f.top) + steps * f.top)
            flops += 2.0 * expert * f.top * (T + steps)
        nbytes += 2.0 * dense * (1 + steps)
        flops += 2.0 * dense * (T + steps)
    places = case["want"] + steps
    return {"bytes": nbytes + 2.0 * head * (1 + steps) + 2.0 * (T + steps) * cfg.width + 4.0 * places * cfg.vocab, "flops": flops + 2.0 * head * places}


def tolerance(case):
    # about four times the largest error against 64 bits that was seen over some hundred drawn cases
    if case["kind"] == "chain" and case["rows"] <= (12 if case["act"] == "f16" else 8):  # 16 bits of fp16 activations, 32 of fp32 ones, beside exact weights
        return {"rel": 1e-4 if case["act"] == "f16" else 1e-5}
    if case["kind"] in ("chain", "gemm"):  # weights and activations rounded to fp16 (Q4_K: its scales and minima too)
        return {"rel": 2.5e-3 if case["fmt"] == "Q4_K" else 1e-3}
    if case["kind"] == "llama":
        return {"rel": 7e-3}
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 4e-3 if case["model"] == "lenesun" else 1.5e-2}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
def _dequant(raw, fmt, N, K):
    _, per, size = FORMATS[fmt]
    b = raw.view(-1, size)
    half = lambda lo: b[:, lo: lo + 2].contiguous().view(torch.float16).double()
    if fmt == "Q8_0":
        w = half(0) * b[:, 2:].contiguous().view(torch.int8).double()
    elif fmt == "Q4_0":
        w = half(0) * (torch.cat([b[:, 2:] & 15, b[:, 2:] >> 4], dim=1).double() - 8.0)
    else:
        s = b[:, 4:16]
        sc = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6 << 4)], dim=1).double()
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | (s[:, 4:8] >> 6 << 4)], dim=1).double()
        q = b[:, 16:].reshape(-1, 4, 32)
        q = torch.stack([q & 15, q >> 4], dim=2).reshape(-1, 8, 32).double()
        w = (half(0) * sc)[:, :, None] * q - (half(2) * mn)[:, :, None]
    return w.reshape(N, K)


def _rms(x, w, eps, groups=1):
    part = x.reshape(*x.shape[:-1], groups, -1)
    return (part * torch.rsqrt(part.square().mean(-1, keepdim=True) + eps)).reshape(x.shape) * w.double()


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt(d.square().mean(-1, keepdim=True) + eps) * w.double()


def _turn(x, base, first=0, halves=False):
    """x [T, heads, n] turned by position: neighbours, or (halves) the elements half a head apart."""
    T, _, n = x.shape
    i = torch.arange(n // 2, dtype=torch.float64, device=x.device)
    ang = torch.arange(first, first + T, dtype=torch.float64, device=x.device)[:, None] * float(base) ** (-2.0 * i / n)[None, :]
    c, s = ang.cos()[:, None, :], ang.sin()[:, None, :]
    a, b = (x[..., : n // 2], x[..., n // 2:]) if halves else (x[..., 0::2], x[..., 1::2])
    y = (a * c - b * s, b * c + a * s)
    return torch.cat(y, dim=-1) if halves else torch.stack(y, dim=-1).reshape(x.shape)


def _attend(q, k, v, scale, window=None, sink=None):
    """Causal attention of [T, heads, .] queries over [T, kv heads, .]; sink: a logit per head without a value."""
    T, H, _ = q.shape
    rep, out = H // k.shape[1], torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    at = torch.arange(T, device=q.device)
    hidden = at[None, :] > at[:, None]
    if window is not None:
        hidden |= at[:, None] - at[None, :] >= window
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].T * scale).masked_fill_(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], dim=1)
        out[:, h] = s.softmax(-1)[:, :T] @ v[:, h // rep]
    return out.reshape(T, -1)


def _exact_llama(case, seed):
    w, tokens = _llama_inputs(case, seed)
    T = case["prompt"] + case["steps"]
    rows = _llama_config(case).max_seq
    H, G, hd = case["heads"], case["kv_heads"], case["head"]
    lin = lambda x, raw, N, K: x @ _dequant(raw, case["fmt"], N, K).T
    x = w["embedding"].double()[torch.from_numpy(tokens[:T]).cuda()]
    caches = {"k": [], "v": []}
    for lw in w["layers"]:
        p = {k: (lw[k], *s) for k, s in _llama_shapes(case).items()}
        qkv = lin(_rms(x, lw["attn_norm"], 1e-5), *p["wqkv"]).reshape(T, H + 2 * G, hd)
        q, k, v = _turn(qkv[:, :H], 10000.0, halves=True), _turn(qkv[:, H: H + G], 10000.0, halves=True), qkv[:, H + G:]
        for n, t in (("k", k), ("v", v)):
            c = torch.zeros((rows, G * hd), dtype=torch.float64, device="cuda")
            c[:T] = t.reshape(T, -1)
            caches[n].append(c)
        x = x + lin(_attend(q, k, v, hd ** -0.5), *p["wo"])
        h = _rms(x, lw["ffn_norm"], 1e-5)
        x = x + lin(torch.nn.functional.silu(lin(h, *p["wgate"])) * lin(h, *p["wup"]), *p["wdown"])
    logits = lin(_rms(x[T - 1:], w["final_norm"], 1e-5), w["lm_head"], case["vocab"], case["hidden"])
    return {"logits": logits[0], **caches}


def _exact_layers(case, seed):
    cfg, w, tokens = _layer_inputs(case, seed)
    T, eps = len(tokens), cfg.norm_eps
    at = torch.tensor(tokens, device="cuda")
    x = w["embed"][at].double() * cfg.embed_scale
    lin = lambda x, d, n: x @ d[n].double().T + (d[n + ".b"].double() if n + ".b" in d else 0.0)
    norm = _layer_norm if cfg.norm_center else lambda v, wt, e: _rms(v, wt, e, cfg.norm_groups)
    if cfg.bigram:
        b = cfg.bigram
        row = torch.cat([torch.tensor([b.buckets], device="cuda"), (at[:-1] * b.mul_prev + at[1:] * b.mul_cur) % b.buckets])
        x = x + w["bigram"][row].double()
    v_first, latents = None, {}
    for i, (l, d) in enumerate(zip(cfg.layers, w["layers"])):
        m, f, mix = l.mixer, l.mlp, d["mix"]
        h = norm(x, d["norm1"], eps)
        if isinstance(m, GatedRecurrence):
            z, u = torch.sigmoid(lin(h, mix, "z")), lin(h, mix, "x")
            c = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
            states, s = torch.empty_like(u), torch.zeros_like(u[0])
            for t in range(T):
                s = torch.lerp(s, c[t], z[t])
                states[t] = s
            y = lin(states * torch.nn.functional.silu(lin(h, mix, "g")), mix, "o")
        elif isinstance(m, WindowAttention):
            q, k, v = (lin(h, mix, n).reshape(T, c, m.dim) for n, c in (("q", m.heads), ("k", m.kv_heads), ("v", m.kv_heads)))
            v_first, v = (v, v) if v_first is None else (v_first, torch.lerp(v, v_first, mix["vmix"]))
            y = lin(_attend(_turn(q, m.rot.base), _turn(k, m.rot.base), v, m.scale, m.window, torch.zeros(m.heads, dtype=torch.float64, device="cuda")),
                    mix, "o")
        else:
            q = lin(_rms(lin(h, mix, "dq"), mix["dq.norm"], eps), mix, "uq").reshape(T, m.heads, -1)
            q = torch.cat([q[..., : m.dim], _turn(q[..., m.dim:], m.rot.base)], dim=-1)
            if m.kv_from is None:
                a = lin(h, mix, "dkv")
                latents[i] = _rms(a[:, : m.kv_rank], mix["dkv.norm"], eps), _turn(a[:, None, m.kv_rank:], m.rot.base)
            c, r = latents[i if m.kv_from is None else m.kv_from]
            k = torch.cat([lin(c, mix, "uk").reshape(T, m.heads, -1), r.expand(-1, m.heads, -1)], dim=-1)
            y = lin(_attend(q, k, lin(c, mix, "uv").reshape(T, m.heads, -1), m.scale, None, mix["sink"].double()), mix, "o")
        if isinstance(f, MixtureOfExperts):  # (beside the mixer)
            e = d["mlp"]
            top, ids = lin(h, e, "router").topk(f.top, dim=-1)
            wt = top.softmax(-1)
            for j in range(f.experts):
                t, k = (ids == j).nonzero(as_tuple=True)
                g, u = (h[t] @ e["gate"][j].double().T).clamp(max=f.limit), (h[t] @ e["up"][j].double().T).clamp(-f.limit, f.limit)
                y.index_add_(0, t, wt[t, k, None] * ((g * torch.sigmoid(f.alpha * g) * (u + f.beta)) @ e["down"][j].double().T))
        if cfg.parallel:
            x = x + cfg.residual_mult * y
            continue
        x = x + norm(y, d["norm1b"], eps)
        if f is not None:
            y = lin(lin(norm(x, d["norm2"], eps), d["mlp"], "up").clamp(min=0.0).square(), d["mlp"], "down")
            x = x + norm(y, d["norm2b"], eps)
    places = x[case["prompt"] - case["want"]:]
    return norm(places, w["final_norm"], eps) @ w["embed" if cfg.tied_head else "head"].double().T


def exact(case, seed):
    if case["kind"] == "llama":
        return _exact_llama(case, seed)
    if case["kind"] == "layers":
        return _exact_layers(case, seed)
    W, A, D = _matmul_inputs(case, seed)
    out = []
    for w, a, d in zip(W, A, D):
        y = a.double() @ _dequant(w, case["fmt"], case["N"], case["K"]).T
        out.append(torch.nn.functional.silu(y) if case["fuse"] == "silu" else y + d.double() if case["fuse"] == "add" else y)
    return out
