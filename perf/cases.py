"""Timing cases of the quantised-matmul engine: what a host runtime asks of it, through the Python API.

A decode step runs the projections of every layer at batch 1, the speculative verifier the same
layers with a few rows, prefill the GEMM on a chunk of the prompt; the lm_head picks the next token
and the embedding table turns it into the next hidden state.  Around that: single projections of any
size, the runner that stages rows from pinned host memory and reads results back, bulk
dequantisation, and the one-shot call on host buffers.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cogni_ml_b200 import (DeviceQuantWeight, GemvMany, Projection, QuantMatmul,
                           QuantProjectionRunner, QuantWeight)

TYPES = {"q8_0": 8, "q4_k": 12, "q5_k": 13, "q6_k": 14, "iq4_nl": 20}
BLOCK = {8: (34, 32), 12: (144, 256), 13: (176, 256), 14: (210, 256), 20: (18, 32)}  # bytes, elements


def listed():
    return [
        # the smallest projection of the configurations: one launch, latency counts
        {"name": "gemv_q8_small", "kind": "gemv", "type": "q8_0", "out": 3584, "in": 1024, "batch": 1, "addend": "none"},
        # a width that no 256-element superblock divides (what Q8_0 / IQ4_NL are chosen for), odd rows, a bias
        {"name": "gemv_ragged", "kind": "gemv", "type": "iq4_nl", "out": 2053, "in": 2976, "batch": 3, "addend": "bias"},
        # one 9B-shaped layer's projections, one token: the decode step
        {"name": "layer_9b_b1", "kind": "layer", "attn": "q4_k", "up": "q4_k", "down": "q6_k",
         "hidden": 4096, "kv": 1024, "ffn": 12288, "batch": 1},
        # one 27B-shaped layer with the speculative verifier's rows
        {"name": "layer_27b_b8", "kind": "layer", "attn": "q5_k", "up": "q4_k", "down": "q6_k",
         "hidden": 5120, "kv": 1024, "ffn": 17408, "batch": 8},
        # the resident runner: rows staged from the host, run, read back
        {"name": "runner_9b_t16", "kind": "runner", "attn": "q4_k", "up": "q4_k", "down": "q6_k",
         "hidden": 4096, "kv": 1024, "ffn": 12288, "batch": 16},
        # output norm -> lm_head -> argmax -> embedding of the chosen token, one row
        {"name": "head_top1_b1", "kind": "head", "type": "q6_k", "vocab": 151936, "dim": 5120, "batch": 1, "top": 1},
        # the verifier's head: the two best tokens of every row
        {"name": "head_top2_b5", "kind": "head", "type": "q6_k", "vocab": 151936, "dim": 4096, "batch": 5, "top": 2},
        # prompt chunks: a short odd one, an ordinary one, the largest
        {"name": "prefill_q5_m77", "kind": "prefill", "type": "q5_k", "m": 77, "n": 4096, "k": 4096, "dtype": "f32"},
        {"name": "prefill_q4_m512", "kind": "prefill", "type": "q4_k", "m": 512, "n": 12288, "k": 4096, "dtype": "f32"},
        {"name": "prefill_q6_m4096", "kind": "prefill", "type": "q6_k", "m": 4096, "n": 4096, "k": 12288, "dtype": "bf16"},
        # a whole tensor to f32
        {"name": "dequant_q6", "kind": "dequant", "type": "q6_k", "out": 4096, "in": 12288},
        # the drop-in call on host arrays, weight bytes included
        {"name": "host_q4", "kind": "host", "type": "q4_k", "out": 4096, "in": 4096, "batch": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, t, lo, hi):
    """A row length that type t can have: whole blocks of it."""
    be = BLOCK[TYPES[t]][1]
    return max(be, _log(rng, lo, hi) // be * be)


def draw(rng):
    kind = rng.choice(("gemv", "gemv", "layer", "layer", "runner", "head", "prefill", "prefill", "dequant", "host"))
    kt = ("q8_0", "q4_k", "q5_k", "q6_k", "iq4_nl")
    t = rng.choice(kt)
    if kind == "gemv":
        return {"kind": kind, "type": t, "out": _log(rng, 64, 24576), "in": _width(rng, t, 512, 16384),
                "batch": rng.randint(1, 16), "addend": rng.choice(("none", "bias", "residual"))}
    if kind in ("layer", "runner"):
        return {"kind": kind, "attn": rng.choice(kt), "up": rng.choice(("q4_k", "q5_k", "q8_0", "iq4_nl")),
                "down": rng.choice(("q6_k", "q5_k", "q8_0", "q4_k")), "hidden": 256 * rng.randint(4, 20),
                "kv": 128 * rng.randint(1, 16), "ffn": 256 * _log(rng, 10, 68), "batch": rng.randint(1, 16)}
    if kind == "head":
        return {"kind": kind, "type": rng.choice(("q6_k", "q4_k", "q8_0")), "vocab": _log(rng, 32000, 151936),
                "dim": 256 * rng.randint(4, 20), "batch": rng.randint(1, 8), "top": rng.choice((1, 2))}
    if kind == "prefill":
        return {"kind": kind, "type": t, "m": _log(rng, 17, 4096), "n": _log(rng, 512, 12288) // 8 * 8,
                "k": 256 * _log(rng, 4, 16), "dtype": rng.choice(("f32", "bf16"))}
    if kind == "dequant":
        return {"kind": kind, "type": t, "out": _log(rng, 64, 12288), "in": _width(rng, t, 1024, 4096)}
    return {"kind": "host", "type": t, "out": _log(rng, 64, 4096), "in": _width(rng, t, 512, 4096), "batch": rng.randint(1, 8)}


# ------------------------------------------------------------------------------------------ inputs
class _Maker:
    """Tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(int(seed))

    def rows(self, *shape):
        return torch.randn(*shape, dtype=torch.float32, device="cuda", generator=self.gen)

    def raw(self, t, out_dim, in_dim):
        """GGUF bytes of an [out_dim, in_dim] weight: uniform quants and sub-block scales, fp16 block
        scales |N(0, s)| of the size trained weights have (weight rms about 0.04)."""
        bb, be = BLOCK[t]
        nb = out_dim * (in_dim // be)
        w = torch.randint(0, 256, (nb, bb), dtype=torch.uint8, device="cuda", generator=self.gen)

        def put(at, sigma):
            d = torch.randn(nb, 1, device="cuda", generator=self.gen).abs_().mul_(sigma)
            w[:, at:at + 2] = d.to(torch.float16).view(torch.uint8)

        if t in (12, 13):
            put(0, 1e-4 if t == 12 else 5e-5)
            put(2, 7.5e-4)
        elif t == 14:
            # the int8 sub-block scales in [-64, 63]
            w[:, 192:208] = torch.randint(-64, 64, (nb, 16), dtype=torch.int8, device="cuda",
                                          generator=self.gen).view(torch.uint8)
            put(208, 6e-5)
        else:
            put(0, 5.5e-4)
        return w.view(-1)

    def device(self, t, out_dim, in_dim):
        w = DeviceQuantWeight(self.raw(t, out_dim, in_dim), t, out_dim, in_dim)
        w.resident = True  # complete before anything that uses it is launched
        return w

    def host(self, t, out_dim, in_dim):
        return QuantWeight(self.raw(t, out_dim, in_dim).cpu().numpy(), t, out_dim, in_dim)

    def norm(self, n):
        return 1.0 + 0.1 * self.rows(n)


def prepare(case, seed):
    mk, kind = _Maker(seed), case["kind"]
    s = {"kind": kind}
    if kind == "gemv":
        n, k, b = case["out"], case["in"], case["batch"]
        s.update(w=mk.device(TYPES[case["type"]], n, k), x=mk.rows(b, k), add={})
        if case["addend"] == "bias":
            s["add"] = {"bias": mk.rows(n)}
        elif case["addend"] == "residual":
            s["add"] = {"residual": mk.rows(b, n)}
    elif kind in ("layer", "runner"):
        h, kv, f, b = case["hidden"], case["kv"], case["ffn"], case["batch"]
        ta, tu, td = TYPES[case["attn"]], TYPES[case["up"]], TYPES[case["down"]]
        if kind == "layer":
            x, new = mk.rows(b, h), lambda n: torch.empty(b, n, dtype=torch.float32, device="cuda")
            qkv, gu, mid = [new(h), new(kv), new(kv)], [new(f), new(f)], new(h)
            s.update(x=x, mid=mid, y=new(h), o=mk.device(ta, h, h), down=mk.device(td, h, f),
                     qkv=GemvMany([mk.device(ta, n, h) for n in (h, kv, kv)], x, qkv, norm_weight=mk.norm(h)),
                     up=GemvMany([mk.device(tu, f, h) for _ in range(2)], mid, gu, norm_weight=mk.norm(h)))
        else:
            ps = [Projection("q", mk.host(ta, h, h), "x"), Projection("k", mk.host(ta, kv, h), "x"),
                  Projection("v", mk.host(ta, kv, h), "x"), Projection("o", mk.host(ta, h, h), "attn", "x"),
                  Projection("gate", mk.host(tu, f, h), "mid"), Projection("up", mk.host(tu, f, h), "mid"),
                  Projection("down", mk.host(td, h, f), "act", "mid")]
            rows = {"x": h, "attn": h, "mid": h, "act": f}
            r = QuantProjectionRunner.from_weights(ps, b, {k: mk.rows(b, n).cpu().numpy() for k, n in rows.items()})
            r.upload_weights()
            s["runner"] = r
    elif kind == "head":
        s.update(w=mk.device(TYPES[case["type"]], case["vocab"], case["dim"]), x=mk.rows(case["batch"], case["dim"]),
                 norm=mk.norm(case["dim"]), top=case["top"])
    elif kind == "prefill":
        s.update(w=mk.device(TYPES[case["type"]], case["n"], case["k"]),
                 x=mk.rows(case["m"], case["k"]).to(torch.bfloat16),
                 dtype=torch.bfloat16 if case["dtype"] == "bf16" else torch.float32)
    elif kind == "dequant":
        s.update(w=mk.device(TYPES[case["type"]], case["out"], case["in"]))
    else:
        w = mk.host(TYPES[case["type"]], case["out"], case["in"])
        s.update(w=w, x=mk.rows(case["batch"], case["in"]).cpu().numpy(), bias=mk.rows(case["out"]).cpu().numpy(),
                 rows=case["batch"])
    return s


# -------------------------------------------------------------------------------------------- runs
def run(s):
    kind = s["kind"]
    if kind == "gemv":
        return s["w"].gemv(s["x"], **s["add"])
    if kind == "layer":
        # attention itself belongs to the host runtime: the rows of q stand for its output
        q, k, v = s["qkv"].run()
        s["o"].gemv(q, out=s["mid"], residual=s["x"])
        gate, up = s["up"].run()
        s["down"].gemv_swiglu(gate, up, out=s["y"], residual=s["mid"])
        return q, k, v, s["mid"], gate, up, s["y"]
    if kind == "runner":
        r = s["runner"]
        r.reset_sequence()
        r.run_sequence()
        return r.read_outputs()
    if kind == "head":
        if s["top"] == 2:
            return s["w"].gemv_top2(s["x"])
        idx, val = s["w"].gemv_top1(s["x"], norm_weight=s["norm"])
        return idx, val, s["w"].embedding_lookup(idx, check_range=False)
    if kind == "prefill":
        return s["w"].gemm(s["x"], out_dtype=s["dtype"])
    if kind == "dequant":
        return s["w"].dequantize()
    w = s["w"]
    return QuantMatmul.matmul_add(s["x"], s["rows"], w.in_dim, w.raw, w.type, w.out_dim, s["bias"])


# ------------------------------------------------------------------------------- work and tolerance
def _wb(t, out_dim, in_dim):
    bb, be = BLOCK[TYPES[t]]
    return out_dim * (in_dim // be) * bb


def work(case):
    kind, b = case["kind"], case.get("batch", 1)
    if kind in ("gemv", "host"):
        n, k = case["out"], case["in"]
        add = {"none": 0, "bias": n, "residual": b * n}[case.get("addend", "bias")]
        return {"bytes": _wb(case["type"], n, k) + 4 * (b * (n + k) + add), "flops": 2 * b * n * k}
    if kind in ("layer", "runner"):
        h, kv, f = case["hidden"], case["kv"], case["ffn"]
        w = _wb(case["attn"], 2 * h + 2 * kv, h) + _wb(case["up"], 2 * f, h) + _wb(case["down"], h, f)
        vals = b * (h + h + 2 * kv + h + 2 * f + h) + 2 * h  # x, q, k, v, mid, gate, up, y and the two norms
        if kind == "runner":
            vals = b * (3 * h + f + h + 2 * kv + h + 2 * f + h)  # the four inputs, the seven outputs
        return {"bytes": w + 4 * vals, "flops": 2 * b * (h * (2 * h + 2 * kv) + 3 * h * f)}
    if kind == "head":
        n, k = case["vocab"], case["dim"]
        out = b * (8 + 4 * k) + b * _wb(case["type"], 1, k) if case["top"] == 1 else 16 * b
        return {"bytes": _wb(case["type"], n, k) + 4 * (b + 1) * k + out, "flops": 2 * b * n * k}
    if kind == "prefill":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": _wb(case["type"], n, k) + 2 * m * k + (2 if case["dtype"] == "bf16" else 4) * m * n,
                "flops": 2 * m * n * k}
    n, k = case["out"], case["in"]
    return {"bytes": _wb(case["type"], n, k) + 4 * n * k, "flops": 2 * n * k}


def tolerance(case):
    kind = case["kind"]
    if kind == "dequant":
        return "exact"
    if kind == "prefill":
        # operands rounded to bf16, f32 sums; a bf16 result is rounded once more (2^-9)
        return {"rel": 5e-3 if case["dtype"] == "bf16" else 2e-3}
    # activations in 15-bit block floating point: steps of 2^-14 of the largest of a group of 16 to
    # 256, about 5e-5 of the rows' rms; two roundings differ by sqrt(2) of that
    if kind == "layer":
        return {"rel": 4e-4}  # chained, and silu(gate) * up has longer tails than its inputs
    if kind == "head":
        return {"rel": 1e-4, "differ": 0.0}
    return {"rel": 1e-4}


# ------------------------------------------------------------------------- the same in 64 bits
_IQ4_NL = (-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113)


def _nibbles(b):
    return b & 15, b >> 4


def _scales_k4(s):
    """The eight 6-bit scales and minimums of [blocks, 12] bytes."""
    lo, hi, top = s[:, 0:4], s[:, 4:8], s[:, 8:12]
    return (torch.cat([lo & 63, (top & 15) | (lo >> 6 << 4)], 1), torch.cat([hi & 63, (top >> 4) | (hi >> 6 << 4)], 1))


def _wide_blocks(t, raw):
    """GGUF blocks [blocks, bytes] -> their weights [blocks, elements] in f64."""
    def half(at):
        return raw[:, at:at + 2].contiguous().view(torch.float16).double()

    nb, b = raw.shape[0], raw.int()
    if t == 8:
        return half(0) * raw[:, 2:34].contiguous().view(torch.int8).double()
    if t == 20:
        lo, hi = _nibbles(b[:, 2:18])
        table = torch.tensor(_IQ4_NL, dtype=torch.float64, device=raw.device)
        return half(0) * table[torch.cat([lo, hi], 1).long()]
    if t in (12, 13):
        sc, mn = (v.double() for v in _scales_k4(b[:, 4:16]))
        lo, hi = _nibbles(b[:, -128:].reshape(nb, 4, 32))
        q = torch.stack([lo, hi], 2).reshape(nb, 8, 32)
        if t == 13:  # sub-block g's fifth bits are bit g of the 32 qh bytes
            bits = torch.arange(8, device=raw.device, dtype=torch.int32).view(1, 8, 1)
            q = q + ((b[:, 16:48].unsqueeze(1) >> bits & 1) << 4)
        return ((half(0) * sc).unsqueeze(2) * q.double() - (half(2) * mn).unsqueeze(2)).reshape(nb, 256)
    lo, hi = _nibbles(b[:, :128].reshape(nb, 2, 64))
    ql = torch.cat([lo, hi], 2).reshape(nb, 2, 4, 32)
    shift = torch.arange(0, 8, 2, device=raw.device, dtype=torch.int32).view(1, 1, 4, 1)
    q = (ql | (b[:, 128:192].reshape(nb, 2, 1, 32) >> shift & 3) << 4) - 32
    sc = raw[:, 192:208].contiguous().view(torch.int8).double() * half(208)
    return (sc.unsqueeze(2) * q.reshape(nb, 16, 16).double()).reshape(nb, 256)


class _Wide:
    def __init__(self, raw, t, out_dim, in_dim):
        self.t, self.n, self.k = t, out_dim, in_dim
        self.raw = raw.view(out_dim, -1)

    def rows(self, at, count):
        return _wide_blocks(self.t, self.raw[at:at + count].reshape(-1, BLOCK[self.t][0])).view(-1, self.k)

    def mul(self, x, add=0.0):
        step = max(1, (1 << 26) // self.k)
        return torch.cat([x.double() @ self.rows(at, step).T for at in range(0, self.n, step)], 1) + add


class _WideMaker(_Maker):
    def device(self, t, out_dim, in_dim):
        return _Wide(self.raw(t, out_dim, in_dim), t, out_dim, in_dim)

    host = device


def exact(case, seed):
    mk, kind = _WideMaker(seed), case["kind"]

    def normed(x, w):
        x = x.double()
        return x * (x.square().mean(1, keepdim=True) + 1e-6).rsqrt() * w.double()

    if kind == "gemv":
        n, k, b = case["out"], case["in"], case["batch"]
        w, x = mk.device(TYPES[case["type"]], n, k), mk.rows(b, k)
        return w.mul(x, {"none": lambda: 0.0, "bias": lambda: mk.rows(n), "residual": lambda: mk.rows(b, n)}[case["addend"]]())
    if kind in ("layer", "runner"):
        h, kv, f, b = case["hidden"], case["kv"], case["ffn"], case["batch"]
        ta, tu, td = TYPES[case["attn"]], TYPES[case["up"]], TYPES[case["down"]]
        if kind == "layer":
            x = mk.rows(b, h)
            wo, wd = mk.device(ta, h, h), mk.device(td, h, f)
            wq, nq = [mk.device(ta, n, h) for n in (h, kv, kv)], mk.norm(h)
            wu, nu = [mk.device(tu, f, h) for _ in range(2)], mk.norm(h)
            q, k, v = [w.mul(normed(x, nq)) for w in wq]
            mid = wo.mul(q, x)
            gate, up = [w.mul(normed(mid, nu)) for w in wu]
            return q, k, v, mid, gate, up, wd.mul(gate * torch.sigmoid(gate) * up, mid)
        names = ("q", "k", "v", "o", "gate", "up", "down")
        ws = [mk.host(t, n, k) for t, n, k in ((ta, h, h), (ta, kv, h), (ta, kv, h), (ta, h, h), (tu, f, h), (tu, f, h), (td, h, f))]
        rows = {name: mk.rows(b, n) for name, n in (("x", h), ("attn", h), ("mid", h), ("act", f))}
        src = ("x", "x", "x", "attn", "mid", "mid", "act")
        add = {"o": rows["x"], "down": rows["mid"]}
        return {name: w.mul(rows[s], add.get(name, 0.0)) for name, w, s in zip(names, ws, src)}
    if kind == "head":
        w, x = mk.device(TYPES[case["type"]], case["vocab"], case["dim"]), mk.rows(case["batch"], case["dim"])
        if case["top"] == 2:
            return None, w.mul(x).topk(2, 1).values
        return None, w.mul(normed(x, mk.norm(case["dim"]))).amax(1), None  # indices: whole values
    if kind == "prefill":
        w = mk.device(TYPES[case["type"]], case["n"], case["k"])
        return w.mul(mk.rows(case["m"], case["k"]).to(torch.bfloat16))
    if kind == "dequant":
        w = mk.device(TYPES[case["type"]], case["out"], case["in"])
        return w.rows(0, w.n)
    w = mk.host(TYPES[case["type"]], case["out"], case["in"])
    x = mk.rows(case["batch"], case["in"])
    return w.mul(x, mk.rows(case["out"])).reshape(-1)
