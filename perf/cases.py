"""The work this library is used for, as a list of cases and a generator of more cases of the same ranges.

Kinds of case, each one pass through public entry points:

  train    lightning_attn_func forward and backward, tensors (b, h, n, dim) contiguous
  block    what an attention block of a model does around its projections: q, k, v as (b, n, h * dim) projection outputs viewed
           in place, lightning_attn_func, srmsnorm_sigmoid_gate on the heads side by side, and the backward of all of it
  prefill  lightning_attn_prefill of one more piece of a sequence onto a carried state
  decode   lightning_attn_decode, one token per sequence, state updated in place
  norm     SimpleRMSNorm forward and backward
  gate     srmsnorm_sigmoid_gate forward and backward
"""
import math

import torch

import lightning_attention_b200 as la
from lightning_attention_b200.ops.cuda.lightning_attn2 import lightning_attn_decode, lightning_attn_prefill
from lightning_attention_b200.ops.cuda.srmsnorm import srmsnorm_sigmoid_gate

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _attn(name, kind, b, h, n, d, e, dtype="bf16", decay=True, scale=1.0):
    return {"name": name, "kind": kind, "b": b, "h": h, "n": n, "d": d, "e": e, "dtype": dtype, "decay": decay, "scale": scale}


def _rows(name, kind, rows, dim, dtype="bf16"):
    return {"name": name, "kind": kind, "rows": rows, "dim": dim, "dtype": dtype}


def listed():
    return [
        # smallest training call: four heads of a toy model, bound by launches and host work
        _attn("train_small", "train", 1, 4, 256, 64, 64),
        # one step of the reference's own shape list: ragged length, fp16, no decay, value width other than key width
        _attn("train_ragged_fp16", "train", 6, 8, 1213, 128, 64, dtype="fp16", decay=False, scale=0.1),
        # the README example: few (batch, head) pairs, a head width above 128 that is no power of two
        _attn("train_readme", "train", 2, 12, 2048, 192, 192),
        # ordinary training step: the benchmark's sweep at a usual context length
        _attn("train_2k", "train", 4, 32, 2048, 128, 128),
        # the sweep's largest point
        _attn("train_32k", "train", 4, 32, 32768, 128, 128),
        # long context on one GPU: few pairs, very long sequences
        _attn("train_131k", "train", 1, 32, 131072, 128, 128, scale=0.5),
        # attention block of a 2048-wide layer in training, fed by its projections
        _attn("block_4k", "block", 2, 16, 4096, 128, 128),
        # serving: the next piece of one prompt, of no round length, onto its carried state
        _attn("prefill_5000", "prefill", 1, 32, 5000, 128, 128, scale=0.5),
        # serving: one token for a single sequence, bound by latency
        _attn("decode_1", "decode", 1, 32, 1, 128, 128),
        # serving: one token for a full batch, bound by the state's bytes
        _attn("decode_256", "decode", 256, 32, 1, 128, 128),
        # normalisation of a training batch's hidden states
        _rows("norm_32768x4096", "norm", 32768, 4096),
        # the norm tests' largest fp32 shape: odd row count, small rows
        _rows("norm_fp32_8200x1024", "norm", 8 * 1025, 1024, dtype="fp32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train"] * 5 + ["block", "prefill", "prefill", "decode", "norm", "gate"])
    if kind in ("norm", "gate"):
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        # model widths, now and then one that is a multiple of 8 only
        dim = rng.choice([256 * rng.randint(2, 32), 8 * rng.randint(64, 640)])
        rows = _log_int(rng, 64, min(65536, (1 << 27) // dim))
        c = _rows("", kind, rows, dim, dtype)
    elif kind == "decode":
        d = rng.choice([64, 64, 96, 128, 128, 192, 256])
        h = rng.choice([8, 12, 16, 32])
        c = _attn("", kind, _log_int(rng, 1, max(2, (1 << 27) // (d * d * h))), h, 1, d, d, rng.choice(["bf16", "bf16", "fp16"]), rng.random() < 0.85)
    else:
        d = rng.choice([64, 64, 80, 96, 128, 128, 128, 192, 256])
        e = d if kind != "train" or d > 128 or rng.random() < 0.8 else rng.choice([64, 128])
        h = rng.choice([4, 8, 12, 16, 20, 32])
        b = rng.choice([1, 2, 4, 6, 8]) if kind != "prefill" else rng.choice([1, 1, 2, 4])
        # at most a quarter of the largest listed case's elements (a sixteenth for wide heads)
        most = (1 << 26 if d > 128 else 1 << 28) // (b * h * (d + e))
        n = _log_int(rng, 128, max(256, min(65536, most)))
        if rng.random() < 0.4:
            n = 128 * max(1, n // 128)
        c = _attn("", kind, b, h, n, d, e, rng.choice(["bf16", "bf16", "fp16"]), rng.random() < 0.75, 0.5)
    del c["name"]
    return c


def _slopes(case):
    return la._build_slope_tensor(case["h"]).to(DEV, torch.float32) if case["decay"] else None


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    dt = DTYPES[case["dtype"]]

    def rnd(shape, scale=1.0, grad=False):
        t = torch.randn(shape, generator=gen, device=DEV, dtype=dt)
        if scale != 1.0:
            t *= scale
        return t.requires_grad_(grad)

    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("norm", "gate"):
        shape = (case["rows"], case["dim"])
        st["x"], st["dy"] = rnd(shape, grad=True), rnd(shape)
        if kind == "norm":
            st["norm"] = la.SimpleRMSNorm(case["dim"])
        else:
            st["gate"] = rnd(shape, grad=True)
        return st
    b, h, n, d, e, sc = (case[x] for x in ("b", "h", "n", "d", "e", "scale"))
    st["s"] = _slopes(case)
    if kind == "decode":
        st["q"], st["k"], st["v"] = rnd((b, h, d)), rnd((b, h, d)), rnd((b, h, e))
        # the spread that the state of a long prompt has: sqrt(sum_j lambda^2j), at most that of 2048 tokens
        s = st["s"].reshape(-1) if case["decay"] else torch.zeros(h, device=DEV)
        spread = torch.sqrt(1.0 / (1.0 - torch.exp(-2.0 * s)).clamp(min=1.0 / 2048)).reshape(1, h, 1, 1)
        st["kv"] = torch.randn((b, h, e, d), generator=gen, device=DEV) * spread
    elif kind == "block":
        st["h"], st["d"] = h, d
        st["q"], st["k"], st["v"] = (rnd((b, n, h * d), sc, True) for _ in range(3))
        st["gate"], st["dy"] = rnd((b, n, h * d), 1.0, True), rnd((b, n, h * d))
    else:
        grad = kind == "train"
        st["q"], st["k"], st["v"] = rnd((b, h, n, d), sc, grad), rnd((b, h, n, d), sc, grad), rnd((b, h, n, e), sc, grad)
        if grad:
            st["do"] = rnd((b, h, n, e), sc)
        else:
            # the state that an earlier piece of the prompt left
            m = 512
            _, st["kv"] = lightning_attn_prefill(rnd((b, h, m, d), sc), rnd((b, h, m, d), sc), rnd((b, h, m, e), sc), st["s"])
    return st


def run(st):
    kind = st["kind"]
    if kind == "train":
        o = la.lightning_attn_func(st["q"], st["k"], st["v"], st["s"])
        dq, dk, dv = torch.autograd.grad(o, (st["q"], st["k"], st["v"]), st["do"])
        return {"o": o, "dq": dq, "dk": dk, "dv": dv}
    if kind == "block":
        h, d = st["h"], st["d"]
        q, k, v = (st[x].view(*st[x].shape[:2], h, d).transpose(1, 2) for x in ("q", "k", "v"))
        o = la.lightning_attn_func(q, k, v, st["s"])
        y = srmsnorm_sigmoid_gate(o.transpose(1, 2).reshape(st["gate"].shape), st["gate"])
        dq, dk, dv, dg = torch.autograd.grad(y, (st["q"], st["k"], st["v"], st["gate"]), st["dy"])
        return {"y": y, "dq": dq, "dk": dk, "dv": dv, "dg": dg}
    if kind == "prefill":
        o, kv = lightning_attn_prefill(st["q"], st["k"], st["v"], st["s"], st["kv"])
        return {"o": o, "kv": kv}
    if kind == "decode":
        o = lightning_attn_decode(st["q"], st["k"], st["v"], st["s"], st["kv"])
        return {"o": o, "kv": st["kv"]}
    if kind == "norm":
        y = st["norm"](st["x"])
        (dx,) = torch.autograd.grad(y, (st["x"],), st["dy"])
        return {"y": y, "dx": dx}
    y = srmsnorm_sigmoid_gate(st["x"], st["gate"])
    dx, dg = torch.autograd.grad(y, (st["x"], st["gate"]), st["dy"])
    return {"y": y, "dx": dx, "dg": dg}


def work(case):
    """Bytes: every input read once, every output written once. Flops of attention: the recurrence itself, 4 d e per token forward
    and 10 d e backward (one of them the state that dq needs again)."""
    size = 4 if case["dtype"] == "fp32" else 2
    kind = case["kind"]
    if kind in ("norm", "gate"):
        el = case["rows"] * case["dim"]
        # norm: x, dy in, y, dx out; gate: x, g, dy in, y, dx, dg out
        return {"bytes": (4 if kind == "norm" else 6) * el * size, "flops": (8 if kind == "norm" else 20) * el}
    b, h, n, d, e = (case[x] for x in ("b", "h", "n", "d", "e"))
    tok = b * h * n
    if kind == "decode":
        return {"bytes": b * h * (8 * d * e + (2 * d + 2 * e) * size), "flops": 5 * tok * d * e}
    if kind == "prefill":
        return {"bytes": tok * (2 * d + 2 * e) * size + 8 * b * h * d * e, "flops": 4 * tok * d * e}
    # train: q, k, v, do in, o, dq, dk, dv out; block: q, k, v, gate, dy in, y, dq, dk, dv, dgate out (o stays inside)
    per = 4 * d + 4 * e if kind == "train" else 10 * d
    return {"bytes": tok * per * size, "flops": 14 * tok * d * e}


def tolerance(case):
    """Four times what the path was measured to differ by from the same computation in 64 bits, worst output of about 60 cases of
    these ranges: attention rounds its in-block scores and the state's tensor-core copy to the 16-bit type once per block (measured
    rel 3.5e-3 bf16, 4.3e-4 fp16; max 7.5e-2, 5.7e-3), the other kinds round their results only (rel 1.7e-3, 2.1e-4, 8.7e-8 in
    fp32; max 3.9e-3, 4.9e-4, 2.1e-6)."""
    dt = case["dtype"]
    if case["kind"] in ("train", "block", "prefill"):
        return {"rel": 1.4e-2, "max": 0.3} if dt == "bf16" else {"rel": 1.7e-3, "max": 2.4e-2}
    return {"bf16": {"rel": 6.7e-3, "max": 1.6e-2}, "fp16": {"rel": 8.4e-4, "max": 2e-3}, "fp32": {"rel": 4e-7, "max": 1e-5}}[dt]
