"""The work that the performance of this library is measured on: quantized weight matmuls as a program that serves a
model issues them, through the library's public Python calls.

Kinds of cases
  layer      the projections of one decoder layer for `tokens` rows of activations: q / k / v as one multi-matrix call with
             the RMSNorm in front, o, gate / up as one multi-matrix call with the RMSNorm in front, down. One row is a
             decode step, 2..8 rows a small batch of sequences, more rows batched decoding, speculation or a prompt.
             `down_type` differs from `type` in the usual mixed files (Q4_K with Q6_K for the down matrix).
  matmul     one matrix.
  moe_token  the expert matmuls of one token: gate / up of its top-k experts on a shared input, down with one input each.
  moe_ffn    router and fused expert FFN for a batch of tokens.
  head       the LM head, with or without the logit soft-cap.
  host       one matrix through the host-pointer call that a CPU program links against (weights registered once, as at
             model load; activations and results in the caller's own memory).

Weights are N(0, 0.02^2) values put into GGUF blocks by plain min / max and absmax quantizers, activations, norm inputs
and router logits are N(0, 1): what the matmuls of a trained model meet, as far as their cost and rounding go.
"""
import math

import numpy as np
import torch

from laplace_b200 import device, matmul
from laplace_b200.ggml import GGMLType, any_row_bytes

EPS = 1e-5


# ---------------------------------------------------------------- the cases

def listed():
    mixed = {"type": "Q4_K", "down_type": "Q6_K"}
    llama = {"hidden": 4096, "kv": 1024, "ffn": 14336}
    return [
        # the smallest call of a decode step: a key or value projection, where launch and latency are all there is
        {"name": "kv_proj_1", "kind": "matmul", "type": "Q4_K", "tokens": 1, "k": 4096, "n": 1024},
        # one decode step of one sequence through the layer of an 8B model in the usual mixed 4-bit file
        {"name": "layer_1", "kind": "layer", "tokens": 1, **llama, **mixed},
        # the same step in an 8-bit file, with a row length that is no power of two
        {"name": "layer_1_q8", "kind": "layer", "tokens": 1, "hidden": 2816, "kv": 1024, "ffn": 8448, "type": "Q8_0", "down_type": "Q8_0"},
        # eight sequences decoded together
        {"name": "layer_8", "kind": "layer", "tokens": 8, **llama, **mixed},
        # a batch of two dozen: batched decoding, or speculated tokens being verified
        {"name": "layer_24", "kind": "layer", "tokens": 24, **llama, **mixed},
        # a short prompt of ragged length in an 8-bit file
        {"name": "layer_77_q8", "kind": "layer", "tokens": 77, "hidden": 2816, "kv": 1024, "ffn": 8448, "type": "Q8_0", "down_type": "Q8_0"},
        # a prompt of 512 tokens: the prefill half of the benchmark
        {"name": "layer_512", "kind": "layer", "tokens": 512, **llama, **mixed},
        # the largest prompt chunk a server would take in one pass
        {"name": "layer_2048", "kind": "layer", "tokens": 2048, **llama, **mixed},
        # one token through the expert matmuls of a mixture-of-experts layer
        {"name": "moe_token", "kind": "moe_token", "type": "Q4_K", "experts": 128, "top_k": 8, "hidden": 2048, "inter": 768},
        # a batch of 256 tokens through router and experts
        {"name": "moe_256", "kind": "moe_ffn", "tokens": 256, "type": "Q4_K", "experts": 128, "top_k": 8, "hidden": 2048, "inter": 768},
        # logits of the next token
        {"name": "head_1", "kind": "head", "type": "Q6_K", "tokens": 1, "hidden": 4096, "vocab": 32000, "softcap": 30.0},
        # the benchmark's matrix through the host-pointer call
        {"name": "host_1", "kind": "host", "type": "Q4_K", "tokens": 1, "k": 4096, "n": 14336},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer"] * 5 + ["matmul"] * 3 + ["moe_token", "moe_ffn", "moe_ffn", "head", "host"])
    if kind == "layer":
        hidden = 256 * rng.randint(4, 16)
        t, d = rng.choice([("Q4_K", "Q6_K"), ("Q4_K", "Q6_K"), ("Q4_K", "Q4_K"), ("Q6_K", "Q6_K"), ("Q8_0", "Q8_0"), ("Q4_0", "Q4_0")])
        return {"kind": kind, "tokens": _log_int(rng, 1, 1500), "hidden": hidden, "kv": 64 * rng.randint(2, 16), "ffn": 256 * rng.randint(hidden // 128, hidden * 7 // 512),
                "type": t, "down_type": d}
    if kind == "matmul":
        t = rng.choice(["Q4_K", "Q4_K", "Q6_K", "Q8_0", "Q4_0", "Q5_0", "Q5_K", "F16"])
        k = (256 if t.endswith("K") else 32) * rng.randint(2, 16) * (1 if t.endswith("K") else rng.choice([1, 8]))
        return {"kind": kind, "type": t, "tokens": rng.choice([1, 1, _log_int(rng, 2, 40)]), "k": k, "n": _log_int(rng, 256, 16384)}
    if kind in ("moe_token", "moe_ffn"):
        e = rng.choice([8, 16, 32, 60, 64, 128])
        c = {"kind": kind, "type": rng.choice(["Q4_K", "Q4_K", "Q6_K", "Q8_0"]), "experts": e, "top_k": rng.randint(2, 8 if e > 8 else 4), "hidden": 256 * rng.randint(4, 10),
             "inter": 256 * rng.randint(2, 6)}
        return dict(c, tokens=_log_int(rng, 2, 600)) if kind == "moe_ffn" else c
    if kind == "head":
        return {"kind": kind, "type": rng.choice(["Q6_K", "Q8_0", "F16", "Q4_K"]), "tokens": rng.choice([1, 1, rng.randint(2, 8)]), "hidden": 256 * rng.randint(4, 16),
                "vocab": rng.randint(16000, 64000), "softcap": rng.choice([0.0, 30.0])}
    return {"kind": kind, "type": rng.choice(["Q4_K", "Q6_K", "Q8_0", "Q4_0"]), "tokens": rng.choice([1, 1, rng.randint(2, 100)]), "k": 256 * rng.randint(4, 16), "n": _log_int(rng, 512, 14336)}


# ------------------------------------------- GGUF blocks, made on the GPU

def _halves(v):
    return v.to(torch.float16).contiguous().view(torch.uint8).reshape(v.shape + (2,))


def _nibbles(q):                                  # [..., 32] -> 16 bytes: value l in the low, l + 16 in the high half of byte l
    return q[..., :16] | (q[..., 16:] << 4)


def _affine32(b, top):
    """Super-blocks [..., 8, 32]: fp16 d and dmin, 6-bit scales and mins, quants 0..top."""
    lo = (-b.amin(-1)).clamp_min(0)
    s, m = (b.amax(-1) + lo) / top, lo
    d, dmin = (s.amax(-1) / 63).half().float(), (m.amax(-1) / 63).half().float()
    sc = (s / d.clamp_min(1e-12)[..., None]).round().clamp(0, 63)
    mn = (m / dmin.clamp_min(1e-12)[..., None]).round().clamp(0, 63)
    step = (d[..., None] * sc).clamp_min(1e-12)
    q = ((b + (dmin[..., None] * mn)[..., None]) / step[..., None]).round().clamp(0, top).to(torch.uint8)
    sc, mn = sc.to(torch.uint8), mn.to(torch.uint8)
    packed = torch.cat([sc[..., :4] | ((sc[..., 4:] >> 4) << 6), mn[..., :4] | ((mn[..., 4:] >> 4) << 6), (sc[..., 4:] & 15) | ((mn[..., 4:] & 15) << 4)], -1)
    return torch.cat([_halves(d), _halves(dmin), packed], -1), q


def _pack_rows(t, w):
    """fp32 rows [N, K] on the GPU -> the rows' GGUF bytes."""
    n, k = w.shape
    if t == "F16":
        return w.half().view(torch.uint8)
    if t in ("Q4_0", "Q5_0", "Q8_0"):
        b = w.view(n, k // 32, 32)
        top = {"Q4_0": 8, "Q5_0": 16, "Q8_0": 127}[t]
        d = (b.abs().amax(-1) / top).half()
        q = (b / d.float().clamp_min(1e-12)[..., None]).round()
        if t == "Q8_0":
            return torch.cat([_halves(d), q.clamp(-127, 127).to(torch.int8).view(torch.uint8)], -1).view(n, -1)
        q = (q + top).clamp(0, 2 * top - 1).to(torch.uint8)
        if t == "Q4_0":
            return torch.cat([_halves(d), _nibbles(q)], -1).view(n, -1)
        bit = (q >> 4).view(n, k // 32, 4, 8) << torch.arange(8, dtype=torch.uint8, device=w.device)
        return torch.cat([_halves(d), bit.sum(-1).to(torch.uint8), _nibbles(q & 15)], -1).view(n, -1)
    if t in ("Q4_K", "Q5_K"):
        head, q = _affine32(w.view(n, k // 256, 8, 32), 15 if t == "Q4_K" else 31)
        low = q & 15
        qs = (low[..., 0::2, :] | (low[..., 1::2, :] << 4)).reshape(n, k // 256, 128)
        if t == "Q4_K":
            return torch.cat([head, qs], -1).view(n, -1)
        high = ((q >> 4) << torch.arange(8, dtype=torch.uint8, device=w.device)[:, None]).sum(-2).to(torch.uint8)
        return torch.cat([head, high, qs], -1).view(n, -1)
    b = w.view(n, k // 256, 16, 16)               # Q6_K
    s = b.abs().amax(-1) / 31
    d = (s.amax(-1) / 127).half()
    sc = (s / d.float().clamp_min(1e-12)[..., None]).round().clamp(-127, 127)
    q = (b / (d.float()[..., None] * sc).clamp_min(1e-12)[..., None]).round().clamp(-32, 31)
    v = (q + 32).to(torch.uint8).view(n, k // 256, 2, 4, 32)
    ql = torch.cat([(v[..., 0, :] & 15) | ((v[..., 2, :] & 15) << 4), (v[..., 1, :] & 15) | ((v[..., 3, :] & 15) << 4)], -1).view(n, k // 256, 128)
    qh = ((v[..., 0, :] >> 4) | ((v[..., 1, :] >> 4) << 2) | ((v[..., 2, :] >> 4) << 4) | ((v[..., 3, :] >> 4) << 6)).view(n, k // 256, 64)
    return torch.cat([ql, qh, sc.to(torch.int8).view(torch.uint8), _halves(d)], -1).view(n, -1)


def _weights(g, t, n, k):
    """A weight matrix as a loader leaves it in GPU memory: the rows' bytes and the slack that the kernels may read."""
    rb = any_row_bytes(GGMLType[t], k)
    out = torch.zeros(n * rb + 64, dtype=torch.uint8, device="cuda")
    rows = out[: n * rb].view(n, rb)
    for r in range(0, n, 8192):                   # in pieces: the fp32 values of a large matrix need not exist at once
        m = min(8192, n - r)
        rows[r:r + m] = _pack_rows(t, torch.randn(m, k, device="cuda", generator=g) * 0.02)
    return out


# ---------------------------------------------------------------- one pass

class _Registered:
    """Host weights registered with the library for as long as this object lives."""

    def __init__(self, data):
        self.data = data
        matmul.matmul_register_weights(data)

    def __del__(self):
        matmul.matmul_unregister_weights(self.data)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind, t = case["kind"], case["type"]
    device.lib()

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    if kind == "layer":
        h, kv, f, m, d = case["hidden"], case["kv"], case["ffn"], case["tokens"], case["down_type"]
        return {"case": case, "x": normal(m, h), "attn": normal(m, h), "mid": normal(m, h), "act": normal(m, f), "norm1": 1 + 0.1 * normal(h), "norm2": 1 + 0.1 * normal(h),
                "qkv": [_weights(g, t, h, h), _weights(g, t, kv, h), _weights(g, t, kv, h)], "o": _weights(g, t, h, h),
                "gate_up": [_weights(g, t, f, h), _weights(g, t, f, h)], "down": _weights(g, d, h, f)}
    if kind == "matmul":
        return {"case": case, "x": normal(case["tokens"], case["k"]), "w": _weights(g, t, case["n"], case["k"])}
    if kind == "head":
        return {"case": case, "x": normal(case["tokens"], case["hidden"]), "w": _weights(g, t, case["vocab"], case["hidden"])}
    if kind == "host":
        w = _weights(g, t, case["n"], case["k"])[:-64].cpu().numpy()
        return {"case": case, "x": normal(case["tokens"], case["k"]).cpu().numpy(), "y": np.empty((case["tokens"], case["n"]), np.float32), "keep": _Registered(w),
                "w": matmul.Tensor(int(GGMLType[t]), w)}
    e, h, i, k = case["experts"], case["hidden"], case["inter"], case["top_k"]
    s = {"case": case, "gate_up": _weights(g, t, e * 2 * i, h), "down": _weights(g, t, e * h, i)}
    if kind == "moe_token":
        s.update(x=normal(1, h), act=normal(k, i), idx=torch.randperm(e, device="cuda", generator=g)[:k].to(torch.int32))
    else:
        s.update(x=normal(case["tokens"], h), logits=normal(case["tokens"], e))
    return s


def run(s):
    c = s["case"]
    kind, t = c["kind"], GGMLType[c["type"]]
    if kind == "layer":
        m, h, kv, f = c["tokens"], c["hidden"], c["kv"], c["ffn"]
        q, k, v = device.gemm_multi(s["x"], s["qkv"], t, m, h, [h, kv, kv], norm_weight=s["norm1"], eps=EPS)
        o = device.gemm(s["attn"], s["o"], t, m, h, h)
        gate, up = device.gemm_multi(s["mid"], s["gate_up"], t, m, h, [f, f], norm_weight=s["norm2"], eps=EPS)
        down = device.gemm(s["act"], s["down"], GGMLType[c["down_type"]], m, f, h)
        return [q, k, v, o, gate, up, down]
    if kind == "matmul":
        return device.gemm(s["x"], s["w"], t, c["tokens"], c["k"], c["n"])
    if kind == "head":
        return device.lm_head(s["x"], s["w"], t, c["tokens"], c["hidden"], c["vocab"], softcap=c["softcap"])
    if kind == "host":
        matmul.matmul_rows(s["x"], s["w"], s["y"], c["tokens"], c["k"], c["n"])
        return s["y"]
    e, h, i, k = c["experts"], c["hidden"], c["inter"], c["top_k"]
    if kind == "moe_token":
        return [device.moe_gemv(s["x"], s["gate_up"], t, s["idx"], h, 2 * i, per_expert_x=False),
                device.moe_gemv(s["act"], s["down"], t, s["idx"], i, h, per_expert_x=True)]
    idx, weight = device.moe_route(s["logits"], k)
    return [idx, weight, device.moe_ffn(s["x"], s["gate_up"], s["down"], t, t, idx, weight, e, h, i, activation=device.SWIGLU)]


# ------------------------------------------------- what a pass cannot do without

def work(case):
    kind = case["kind"]

    def mm(t, m, k, n):                            # (bytes, flops) of one matrix: packed weights, results
        return n * any_row_bytes(GGMLType[t], k) + 4 * m * n, 2 * m * k * n

    if kind == "layer":
        h, kv, f, m, t = case["hidden"], case["kv"], case["ffn"], case["tokens"], case["type"]
        parts = [mm(t, m, h, h), mm(t, m, h, kv), mm(t, m, h, kv), mm(t, m, h, h), mm(t, m, h, f), mm(t, m, h, f), mm(case["down_type"], m, f, h), (4 * m * (3 * h + f) + 8 * h, 0)]
    elif kind in ("matmul", "host"):
        parts = [mm(case["type"], case["tokens"], case["k"], case["n"]), (4 * case["tokens"] * case["k"], 0)]
    elif kind == "head":
        parts = [mm(case["type"], case["tokens"], case["hidden"], case["vocab"]), (4 * case["tokens"] * case["hidden"], 0)]
    else:
        e, h, i, k, t = case["experts"], case["hidden"], case["inter"], case["top_k"], case["type"]
        m = case.get("tokens", 1)
        touched = e * (1 - (1 - k / e) ** m)       # experts that at least one token chooses, on average over the routings
        weights = touched * (2 * i * any_row_bytes(GGMLType[t], h) + h * any_row_bytes(GGMLType[t], i))
        rows = 4 * m * (2 * h + e + 2 * k) if kind == "moe_ffn" else 4 * (h + k * (3 * i + h) + k)
        parts = [(weights + rows, 2 * m * k * 3 * h * i)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """Four times what the path shows against the same sums in 64 bits (listed and drawn cases, two seeds each)."""
    if case["kind"] in ("layer", "moe_ffn"):
        # The activations of the RMSNorm and of the gated activation are quantized to int8 after a 32-bit reduction: one that
        # lies on a rounding boundary moves by a whole step when the reduction's order changes. Seen: 2.5e-4 and 3.0e-3
        # (single rows of 1024 to 3328 values, where one such step weighs most), 1.1e-4 and below for larger cases.
        return {"rel": 1e-3, "max": 1.2e-2}
    return {"rel": 3e-6, "max": 1.2e-5}            # seen: 8e-7 and 3e-6


# ------------------------------------------------- the same results in 64 bits

def _half_at(b, i):                               # fp16 at byte i of every block [..., bytes]
    return b[..., i:i + 2].contiguous().view(torch.float16)[..., 0].double()


def _unpack_nibbles(q):                           # the inverse of _nibbles
    return torch.cat([q & 15, q >> 4], -1)


def _unpack_rows(t, raw, n, k):
    """The values of n rows' GGUF bytes, in 64 bits."""
    rb = any_row_bytes(GGMLType[t], k)
    raw = raw[: n * rb].view(n, rb)
    if t == "F16":
        return raw.view(torch.float16).double()
    if t in ("Q4_0", "Q5_0", "Q8_0"):
        b = raw.view(n, k // 32, -1)
        if t == "Q8_0":
            q = b[..., 2:].contiguous().view(torch.int8).double()
        elif t == "Q4_0":
            q = _unpack_nibbles(b[..., 2:]).double() - 8
        else:
            bit = (b[..., 2:6, None] >> torch.arange(8, dtype=torch.uint8, device=raw.device)) & 1
            q = (_unpack_nibbles(b[..., 6:]) | (bit.reshape(n, k // 32, 32) << 4)).double() - 16
        return (_half_at(b, 0)[..., None] * q).view(n, k)
    b = raw.view(n, k // 256, -1)
    if t == "Q6_K":
        ql, qh = b[..., :128].reshape(n, k // 256, 2, 2, 32), b[..., 128:192].reshape(n, k // 256, 2, 32)
        low = torch.cat([ql & 15, ql >> 4], -2)
        high = torch.stack([(qh >> (2 * i)) & 3 for i in range(4)], -2)
        q = (low | (high << 4)).double() - 32
        sc = b[..., 192:208].contiguous().view(torch.int8).double()
        return (_half_at(b, 208)[..., None, None] * sc[..., None] * q.reshape(n, k // 256, 16, 16)).view(n, k)
    s = b[..., 4:16]                              # Q4_K, Q5_K
    sc = torch.cat([s[..., :4] & 63, (s[..., 8:] & 15) | ((s[..., :4] >> 6) << 4)], -1).double()
    mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1).double()
    qs = b[..., -128:].reshape(n, k // 256, 4, 32)
    q = torch.stack([qs & 15, qs >> 4], -2).reshape(n, k // 256, 8, 32)
    if t == "Q5_K":
        high = (b[..., None, 16:48] >> torch.arange(8, dtype=torch.uint8, device=raw.device)[:, None]) & 1
        q = q | (high << 4)
    return (_half_at(b, 0)[..., None, None] * sc[..., None] * q.double() - (_half_at(b, 2)[..., None] * mn)[..., None]).view(n, k)


def _seen(t, x):
    """Activations as the matmul of weight type t sees them: rounded to 8 bits per 32 values, or as they are."""
    if t in ("F16", "Q5_K"):
        return x.double()
    b = x.float().view(*x.shape[:-1], -1, 32)
    d = b.abs().amax(-1, keepdim=True) / 127
    q = (b * torch.where(d > 0, 1 / d, d)).round()
    return (d.double() * q.double()).view(x.shape)


def exact(case, seed):
    """What run() returns, in 64 bits except for the rounding of the activations to 8 bits, which the path prescribes in 32."""
    s = prepare(case, seed)
    kind, t = case["kind"], case["type"]

    def mm(x, raw, t, k, n):
        x = _seen(t, x)
        return torch.cat([x @ _unpack_rows(t, raw[r * any_row_bytes(GGMLType[t], k):], min(4096, n - r), k).T for r in range(0, n, 4096)], -1)

    if kind == "layer":
        h, kv, f = case["hidden"], case["kv"], case["ffn"]

        def norm(x, w):
            inv = (1 / (x.double().square().mean(-1, keepdim=True) + EPS).sqrt()).float()
            return x * inv * w

        a, b = norm(s["x"], s["norm1"]), norm(s["mid"], s["norm2"])
        return ([mm(a, w, t, h, n) for w, n in zip(s["qkv"], (h, kv, kv))] + [mm(s["attn"], s["o"], t, h, h)] +
                [mm(b, w, t, h, f) for w in s["gate_up"]] + [mm(s["act"], s["down"], case["down_type"], f, h)])
    if kind == "matmul":
        return mm(s["x"], s["w"], t, case["k"], case["n"])
    if kind == "head":
        y, cap = mm(s["x"], s["w"], t, case["hidden"], case["vocab"]), case["softcap"]
        return cap * (y / cap).tanh() if cap else y
    if kind == "host":
        return mm(torch.from_numpy(s["x"]), torch.from_numpy(s["w"].data.reshape(-1)), t, case["k"], case["n"]).numpy()
    e, h, i, k = case["experts"], case["hidden"], case["inter"], case["top_k"]
    gu_bytes, dn_bytes = 2 * i * any_row_bytes(GGMLType[t], h), h * any_row_bytes(GGMLType[t], i)
    gate_up, down = (lambda x, j: mm(x, s["gate_up"][j * gu_bytes:], t, h, 2 * i)), (lambda x, j: mm(x, s["down"][j * dn_bytes:], t, i, h))
    if kind == "moe_token":
        chosen = s["idx"].tolist()
        return [torch.cat([gate_up(s["x"], j) for j in chosen]), torch.cat([down(s["act"][n:n + 1], j) for n, j in enumerate(chosen)])]
    weight, idx = s["logits"].double().softmax(-1).topk(k)
    weight = weight / weight.sum(-1, keepdim=True)
    out = torch.zeros(case["tokens"], h, dtype=torch.float64, device="cuda")
    for j in range(e):
        token, slot = (idx == j).nonzero(as_tuple=True)
        if len(token):
            gate, up = gate_up(s["x"][token], j).split(i, -1)
            out.index_add_(0, token, weight[token, slot, None] * down(torch.nn.functional.silu(gate) * up, j))
    return [None, weight, out]
