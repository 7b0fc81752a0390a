"""Performance cases of the library: the calls that a program holding large
integers makes, over the range of sizes it makes them in.

A case names an operation and its sizes in 64-bit limbs.  Operands are uniform
random limbs with a nonzero top limb (a set top bit for divisors), the
distribution of the library's own benchmark; they sit on the GPU, as do the
results, except for the host drop-in, which takes and fills host arrays."""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import simd_bigint_b200 as sbg
from simd_bigint_b200.workloads import division_shapes, mixed_batch_shapes

# Operands inside one buffer start at multiples of this many limbs, as
# separately allocated ones would.
ALIGN = 64

_ctx = None


def context() -> sbg.Context:
    """The one context a program keeps: its stream, tables and workspace."""
    global _ctx
    if _ctx is None:
        _ctx = sbg.Context(0)
    return _ctx


def listed() -> list[dict]:
    return [
        # a product of two numbers of a few thousand bits: launch latency
        {"name": "mul_40x60", "op": "mul", "an": 60, "bn": 40},
        # a product whose transform one CTA holds (100,000 bits)
        {"name": "mul_1500", "op": "mul", "an": 1500, "bn": 1500},
        # the balanced million-bit product of the CPU-sized configuration
        {"name": "mul_16384", "op": "mul", "an": 16384, "bn": 16384},
        # an odd-sized, unbalanced product, as inside a product tree
        {"name": "mul_333333x77777", "op": "mul", "an": 333333, "bn": 77777},
        # a large square, as inside an exponentiation or a square root
        {"name": "sqr_2p22", "op": "sqr", "an": 1 << 22},
        # the largest balanced product (a billion bits each)
        {"name": "mul_2p24", "op": "mul", "an": 1 << 24, "bn": 1 << 24},
        # a large unbalanced product
        {"name": "mul_2p24x2p20", "op": "mul", "an": 1 << 24, "bn": 1 << 20},
        # the middle product of a Newton step
        {"name": "mulmid_400001x200003", "op": "mulmid", "an": 400001, "bn": 200003},
        # a batch of uneven products, planned once and replayed as a graph
        {"name": "batch_1024", "op": "batch", "count": 1024, "shapes": 12345},
        # a batch of uneven divisions of 2n by n limbs
        {"name": "div_128", "op": "div", "count": 128, "shapes": 4242},
        # one large reciprocal
        {"name": "recip_100000", "op": "recip", "an": 100000},
        # the reference-signature drop-in on host arrays, copies included
        {"name": "host_250000x200000", "op": "host", "an": 250000, "bn": 200000},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng: random.Random) -> dict:
    op = rng.choice(["mul", "mul", "mul", "sqr", "mulmid", "batch", "div", "recip", "host"])
    if op == "mul":
        an = _log(rng, 40, 1 << 24)
        return {"op": op, "an": an, "bn": max(1, int(an / math.exp(rng.uniform(0, math.log(16)))))}
    if op == "sqr":
        return {"op": op, "an": _log(rng, 40, 1 << 24)}
    if op == "mulmid":
        bn = _log(rng, 256, 1 << 21)
        return {"op": op, "an": int(bn * rng.uniform(1.1, 3.0)), "bn": bn}
    if op == "batch":
        return {"op": op, "count": _log(rng, 16, 768), "shapes": rng.randrange(1 << 20)}
    if op == "div":
        return {"op": op, "count": _log(rng, 4, 80), "shapes": rng.randrange(1 << 20)}
    if op == "recip":
        return {"op": op, "an": _log(rng, 128, 1 << 19)}
    an = _log(rng, 1000, 1 << 19)
    return {"op": op, "an": an, "bn": max(1, int(an / math.exp(rng.uniform(0, math.log(4)))))}


def _operands(sizes: list[int], seed: int, top_bit: bool = False) -> tuple[torch.Tensor, list[int]]:
    """One buffer of random limbs on the GPU, and where in it each operand of
    `sizes` limbs starts; every top limb is nonzero (top bit set if asked)."""
    starts, at = [], 0
    for n in sizes:
        starts.append(at)
        at += -(-n // ALIGN) * ALIGN
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (at,), dtype=torch.int64, device="cuda", generator=g)
    tops = torch.tensor([s + n - 1 for s, n in zip(starts, sizes)], device="cuda")
    x[tops] |= -(1 << 63) if top_bit else 1
    return x, starts


def _room(sizes: list[int]) -> tuple[torch.Tensor, list[int]]:
    """A zeroed result buffer and where each result of `sizes` limbs starts."""
    starts, at = [], 0
    for n in sizes:
        starts.append(at)
        at += -(-n // ALIGN) * ALIGN
    return torch.zeros(at, dtype=torch.int64, device="cuda"), starts


def _batch_shapes(case: dict) -> list[tuple[int, int, int]]:
    return mixed_batch_shapes(case["count"], seed=case["shapes"])


def _div_shapes(case: dict) -> list[int]:
    return division_shapes(case["count"], seed=case["shapes"])


def prepare(case: dict, seed: int) -> dict:
    op, ctx = case["op"], context()
    s = {"op": op, "ctx": ctx}
    if op in ("mul", "mulmid"):
        an, bn = case["an"], case["bn"]
        x, (i, j) = _operands([an, bn], seed)
        s.update(a=x[i:i + an], b=x[j:j + bn],
                 r=torch.zeros(an + bn if op == "mul" else an - bn + 3, dtype=torch.int64, device="cuda"))
    elif op == "sqr":
        x, _ = _operands([case["an"]], seed)
        s.update(a=x[:case["an"]], r=torch.zeros(2 * case["an"], dtype=torch.int64, device="cuda"))
    elif op == "recip":
        x, _ = _operands([case["an"]], seed, top_bit=True)
        s.update(a=x[:case["an"]], r=torch.zeros(case["an"], dtype=torch.int64, device="cuda"))
    elif op == "host":
        an, bn = case["an"], case["bn"]
        x, (i, j) = _operands([an, bn], seed)
        h = x.cpu().numpy().view(np.uint64)
        s.update(a=h[i:i + an].copy(), b=h[j:j + bn].copy(), r=np.zeros(an + bn, dtype=np.uint64))
    elif op == "batch":
        shapes = _batch_shapes(case)
        sizes = [n for kind, an, bn in shapes for n in ((an,) if kind == sbg.JOB_SQR else (an, bn))]
        x, at = _operands(sizes, seed)
        r, rat = _room([sbg.out_limbs(*sh) for sh in shapes])
        base, rbase, k, jobs = x.data_ptr(), r.data_ptr(), 0, []
        for (kind, an, bn), ro in zip(shapes, rat):
            pa = base + 8 * at[k]
            pb = pa if kind == sbg.JOB_SQR else base + 8 * at[k + 1]
            k += 1 if kind == sbg.JOB_SQR else 2
            jobs.append((kind, rbase + 8 * ro, pa, pb, an, bn))
        torch.cuda.synchronize()
        batch = sbg.Batch(ctx, jobs)
        batch.capture()
        s.update(x=x, r=r, batch=batch)
    elif op == "div":
        ns = _div_shapes(case)
        x, xat = _operands([2 * n for n in ns], seed)
        d, dat = _operands(ns, seed + (1 << 32), top_bit=True)
        q, qat = _room([n + 1 for n in ns])
        r, rat = _room(ns)
        jobs = [(q.data_ptr() + 8 * qo, r.data_ptr() + 8 * ro, x.data_ptr() + 8 * xo, d.data_ptr() + 8 * do,
                 2 * n, n) for n, qo, ro, xo, do in zip(ns, qat, rat, xat, dat)]
        s.update(x=x, d=d, q=q, r=r, jobs=jobs)
    return s


def run(s: dict):
    op, ctx = s["op"], s["ctx"]
    if op == "mul":
        ctx.mul(s["r"], s["a"], s["b"])
    elif op == "sqr":
        ctx.sqr(s["r"], s["a"])
    elif op == "mulmid":
        ctx.mulmid(s["r"], s["a"], s["b"])
    elif op == "recip":
        ctx.recip(s["r"], s["a"])
    elif op == "batch":
        s["batch"].run()
    elif op == "div":
        ctx.divrem_batch(s["jobs"])
        return s["q"], s["r"]
    else:
        sbg.nt_mul(s["r"], s["a"], len(s["a"]), s["b"], len(s["b"]))
        return s["r"].view(np.int64)
    return s["r"]


def work(case: dict) -> dict:
    """Operand limbs in, result limbs out, 8 bytes each, once; no floating point."""
    op = case["op"]
    if op in ("mul", "host"):
        limbs = 2 * (case["an"] + case["bn"])
    elif op == "sqr":
        limbs = 3 * case["an"]
    elif op == "mulmid":
        limbs = 2 * case["an"] + 3
    elif op == "recip":
        limbs = 2 * case["an"]
    elif op == "batch":
        limbs = sum((an if kind == sbg.JOB_SQR else an + bn) + sbg.out_limbs(kind, an, bn)
                    for kind, an, bn in _batch_shapes(case))
    else:
        limbs = sum(5 * n + 1 for n in _div_shapes(case))
    return {"bytes": 8 * limbs, "flops": 0}


# Python's own integers are exact; past these sizes they take too long.
EXACT_LIMBS = 40000


def _int(x) -> int:
    h = x.cpu().numpy() if isinstance(x, torch.Tensor) else x
    return int.from_bytes(np.ascontiguousarray(h).view("<u8").tobytes(), "little")


def _limbs(v: int, n: int) -> np.ndarray:
    return np.frombuffer(v.to_bytes(8 * n, "little"), dtype="<i8").copy()


def exact(case: dict, seed: int):
    op = case["op"]
    if op not in ("mul", "sqr", "recip", "host") or case["an"] + case.get("bn", case["an"]) > EXACT_LIMBS:
        return None
    if op in ("mul", "host"):
        an, bn = case["an"], case["bn"]
        x, (i, j) = _operands([an, bn], seed)
        return _limbs(_int(x[i:i + an]) * _int(x[j:j + bn]), an + bn)
    n = case["an"]
    x, _ = _operands([n], seed, top_bit=op == "recip")
    v = _int(x[:n])
    if op == "sqr":
        return _limbs(v * v, 2 * n)
    return _limbs(((1 << (128 * n)) - 1) // v - (1 << (64 * n)), n)
