"""Timed cases of the packed-vector ops: what a program that codes shards asks of this library.

A case is one of six kinds of work, each through the public entry points of `fgf_b200.ops` or `fgf_b200.batch`:

  matrix       k source shards -> m rows with a prepared plan or raw coefficients (`dot_product_matrix[_with]` when
               op is "dot", `mul_add_matrix[_with]` when "add"): RS encode, and the accumulating update of parity
  row          the single-row family with raw coefficients: "axpy" (mul_add), "scatter" (one source into m rows)
               and "gather" (k sources into one row)
  encode       a batch of equal stripes sharing one plan, one submission
  rebuild      a batch of equal stripes, four erased shards each at its own positions, decode plan per stripe,
               rebuilt into the shards' own places
  uneven       a batch of stripes of mixed field, k, m and length, one submission
  elementwise  the product of two vectors

Sizes follow bench.py and its configurations. Sources are separate buffers ("apart") or the consecutive shards of
one buffer ("together", a file cut into k pieces, whose offsets are odd when the shard length is).
"""
import math
import random

import torch

from fgf_b200 import batch, codes, ops
from fgf_b200.fields import FIELDS

GF8B, GF8D, GF16, GF32, FP8, FP16, FP32, GF64, FP64 = range(9)
MIB = 1 << 20


def listed():
    return [
        # one small stripe, the latency of a single call: RS(10,4) over GF(2^8)/0x11D, 64 KiB shards
        {"name": "stripe_gf8d_10_4_64k", "kind": "matrix", "field": GF8D, "k": 10, "m": 4, "len": 65536, "op": "dot",
         "raw": False, "layout": "apart"},
        # an AXPY with a raw coefficient on a moderate buffer, as a network-coding recoder calls it
        {"name": "axpy_gf8d_4m", "kind": "row", "field": GF8D, "op": "axpy", "k": 1, "m": 1, "len": 4 * MIB},
        # one large object: RS(10,4), 16 MiB shards
        {"name": "object_gf8d_10_4_16m", "kind": "matrix", "field": GF8D, "k": 10, "m": 4, "len": 16 * MIB,
         "op": "dot", "raw": False, "layout": "apart"},
        # a file cut into 12 consecutive shards whose length is no multiple of 16
        {"name": "file_gf8d_12_4_ragged", "kind": "matrix", "field": GF8D, "k": 12, "m": 4, "len": 1000003,
         "op": "dot", "raw": False, "layout": "together"},
        # the serving shapes: 64 stripes of 1 MiB shards, encoded, and rebuilt with four erasures each
        {"name": "encode_gf8d_10_4_64x1m", "kind": "encode", "field": GF8D, "k": 10, "m": 4, "len": MIB, "stripes": 64},
        {"name": "rebuild_gf8d_10_4_64x1m", "kind": "rebuild", "field": GF8D, "k": 10, "m": 4, "len": MIB,
         "stripes": 64},
        # stripes of many geometries in one submission: k 4..32, m 1..8, shards of 4 KiB to 4 MiB, Gf8D or Gf16
        {"name": "uneven_256", "kind": "uneven", "stripes": 256, "maxlen": 4 * MIB, "geometry": 3},
        # the wide codes: more sources and rows, and the 2- and 4-byte towers
        {"name": "wide_gf16_32_8_16m", "kind": "matrix", "field": GF16, "k": 32, "m": 8, "len": 16 * MIB, "op": "dot",
         "raw": False, "layout": "apart"},
        {"name": "wide_gf32_16_4_8m", "kind": "matrix", "field": GF32, "k": 16, "m": 4, "len": 8 * MIB, "op": "dot",
         "raw": False, "layout": "apart"},
        {"name": "wide_gf8b_64_16_4m", "kind": "matrix", "field": GF8B, "k": 64, "m": 16, "len": 4 * MIB, "op": "dot",
         "raw": False, "layout": "apart"},
        # RS(10,4) over GF(2^64)
        {"name": "object_gf64_10_4_16m", "kind": "matrix", "field": GF64, "k": 10, "m": 4, "len": 16 * MIB,
         "op": "dot", "raw": False, "layout": "apart"},
        # the products of two vectors of 16-bit elements
        {"name": "elementwise_gf16_64m", "kind": "elementwise", "field": GF16, "len": 64 * MIB},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _whole(n, width):
    return max(width, n - n % width)


def draw(rng):
    kind = rng.choice(["matrix", "matrix", "matrix", "matrix", "row", "encode", "rebuild", "uneven", "elementwise"])
    if kind == "uneven":
        return {"kind": kind, "stripes": _log(rng, 16, 256), "maxlen": _log(rng, MIB // 4, 4 * MIB),
                "geometry": rng.randint(4, 1 << 30)}
    if kind in ("encode", "rebuild"):
        # whole sizes of 4 KiB and up, as an object store cuts its stripes
        n = 4096 * _log(rng, 1, 512)
        k, m = rng.randint(4, 14), rng.randint(2, 4)
        most = max(2, (768 * MIB) // (n * (k + m)))
        return {"kind": kind, "field": rng.choice([GF8B, GF8D]), "k": k, "m": m, "len": n,
                "stripes": _log(rng, 2, min(256, most))}
    field = rng.choice([GF8D, GF8D, GF8D, GF8B, GF16, GF16, GF32, GF64, FP8, FP16, FP32, FP64])
    width = FIELDS[field].BYTES
    if kind == "elementwise":
        return {"kind": kind, "field": field, "len": _whole(_log(rng, 65536, 64 * MIB // (4 if width == 8 else 1)), width)}
    if kind == "row":
        while width == 8:  # raw coefficients are 32-bit; the 8-byte fields go through plans
            field = rng.choice([GF8D, GF8B, GF16, GF32])
            width = FIELDS[field].BYTES
        op = rng.choice(["axpy", "scatter", "gather"])
        return {"kind": kind, "field": field, "op": op, "k": rng.randint(2, 8) if op == "gather" else 1,
                "m": rng.randint(2, 8) if op == "scatter" else 1, "len": _whole(_log(rng, 4096, 32 * MIB), width)}
    most_k, most_m = {1: (64, 16), 2: (32, 8), 4: (16, 4), 8: (10, 4)}[width]
    k = rng.randint(2, most_k) if rng.random() < 0.5 else rng.randint(4, min(16, most_k))
    m = rng.randint(1, most_m) if rng.random() < 0.5 else rng.randint(1, 4)
    layout = rng.choice(["apart", "together"])
    n = min(_log(rng, 4096, 16 * MIB), (512 * MIB) // k, (2048 * MIB) // (k * m * width))
    if layout == "together":
        n = min(n, 64 * MIB // k)
    n = _whole(n, width) if rng.random() < 0.4 else n - n % 256  # ragged lengths among even ones
    return {"kind": kind, "field": field, "k": k, "m": m, "len": n, "op": rng.choice(["dot", "dot", "add"]),
            "raw": width < 8 and rng.random() < 0.2, "layout": layout}


def _noise(gen, n):
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=gen)


def _coeffs(rng, field, n):
    top = (1 << (8 * FIELDS[field].BYTES)) - 1
    return [rng.randint(1, top) for _ in range(n)]


def _pieces(buf, n, count):
    return [buf[t * n:(t + 1) * n] for t in range(count)]


def _geometry(case):
    """(field, k, m, length) of each stripe of a mixed submission."""
    rng = random.Random(case["geometry"])
    for _ in range(case["stripes"]):
        field = rng.choice([GF8D, GF16])
        k, m = rng.randint(4, 32), rng.randint(1, 8)
        yield field, k, m, _whole(_log(rng, 4096, case["maxlen"]), FIELDS[field].BYTES)


def _cauchy_plan(field, k, m):
    c = codes.cauchy_matrix(FIELDS[field], m, k)
    return c, ops.Plan.matrix(FIELDS[field], k, m, [c[i][t] for t in range(k) for i in range(m)])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "elementwise":
        n = case["len"]
        return {"kind": kind, "field": FIELDS[case["field"]], "a": _noise(gen, n), "b": _noise(gen, n),
                "out": torch.zeros(n, dtype=torch.uint8, device="cuda")}
    if kind == "row":
        n, k, m = case["len"], case["k"], case["m"]
        return {"kind": kind, "op": case["op"], "field": FIELDS[case["field"]], "len": n,
                "coeffs": [max(2, c) for c in _coeffs(rng, case["field"], max(k, m))],
                "srcs": [_noise(gen, n) for _ in range(k)], "out": _noise(gen, m * n)}
    if kind == "matrix":
        n, k, m, field = case["len"], case["k"], case["m"], case["field"]
        if case["layout"] == "together":
            srcs = _pieces(_noise(gen, k * n), n, k)
        else:
            srcs = [_noise(gen, n) for _ in range(k)]
        vals = _coeffs(rng, field, k * m)
        s = {"kind": kind, "op": case["op"], "raw": case["raw"], "field": FIELDS[field], "len": n, "m": m,
             "srcs": srcs, "out": _noise(gen, m * n)}
        if case["raw"]:
            s["terms"] = [(vals[t * m:(t + 1) * m], srcs[t]) for t in range(k)]
        else:
            s["plan"] = ops.Plan.matrix(FIELDS[field], k, m, vals)
        return s
    jobs = []
    if kind == "uneven":
        shapes, total = [], 0
        for field, k, m, n in _geometry(case):
            step = -(-n // 256) * 256  # a shard starts at a whole 256 bytes, parity rows follow one another
            shapes.append((field, k, m, n, total, step))
            total += k * step + -(-n * m // 256) * 256
        arena = _noise(gen, total)
        plans = {}
        for field, k, m, n, at, step in shapes:
            if (field, k, m) not in plans:
                plans[field, k, m] = _cauchy_plan(field, k, m)[1]
            srcs = [arena[at + t * step:at + t * step + n] for t in range(k)]
            jobs.append(batch.Job(plans[field, k, m], srcs, arena[at + k * step:at + k * step + n * m], n, m))
    else:
        field, k, m, n = case["field"], case["k"], case["m"], case["len"]
        c, plan = _cauchy_plan(field, k, m)
        arena = _noise(gen, case["stripes"] * (k + m) * n)
        plans = {}
        for i in range(case["stripes"]):
            code = arena[i * (k + m) * n:(i + 1) * (k + m) * n]
            shards = _pieces(code, n, k + m)
            if kind == "encode":
                jobs.append(batch.Job(plan, shards[:k], code[k * n:], n, m))
                continue
            lost = tuple(sorted(rng.sample(range(k + m), min(4, m))))
            left = [s for s in range(k + m) if s not in lost][:k]
            if lost not in plans:
                plans[lost] = codes.decode_plan(FIELDS[field], c, left, list(lost))
            jobs.append(batch.Job(plans[lost], [shards[s] for s in left], code, n, len(lost), True,
                                  [e * n for e in lost]))
    runner = batch.Batch()
    return {"kind": kind, "batch": runner, "jobs": runner.prepare(jobs), "out": arena}


def run(state):
    kind = state["kind"]
    if kind == "matrix":
        out, n, m = state["out"], state["len"], state["m"]
        if state["raw"]:
            (ops.dot_product_matrix if state["op"] == "dot" else ops.mul_add_matrix)(state["field"], out, n, m,
                                                                                     state["terms"])
        else:
            (ops.dot_product_matrix_with if state["op"] == "dot" else ops.mul_add_matrix_with)(
                out, n, m, state["plan"], state["srcs"])
        return out
    if kind == "row":
        f, out, c, srcs = state["field"], state["out"], state["coeffs"], state["srcs"]
        if state["op"] == "axpy":
            ops.mul_add(f, out, c[0], srcs[0])
        elif state["op"] == "scatter":
            ops.mul_add_scatter(f, out, state["len"], c, srcs[0])
        else:
            ops.mul_add_gather(f, out, c, srcs)
        return out
    if kind == "elementwise":
        ops.mul_elementwise(state["field"], state["out"], state["a"], state["b"])
        return state["out"]
    state["batch"].run_prepared(state["jobs"])
    return state["out"]


def work(case):
    kind = case["kind"]
    if kind == "elementwise":
        n = 3 * case["len"]
    elif kind == "row":
        n = (case["k"] + 2 * case["m"]) * case["len"]
    elif kind == "matrix":
        n = (case["k"] + case["m"] * (2 if case["op"] == "add" else 1)) * case["len"]
    elif kind == "encode":
        n = case["stripes"] * (case["k"] + case["m"]) * case["len"]
    elif kind == "rebuild":
        n = case["stripes"] * (case["k"] + min(4, case["m"])) * case["len"]
    else:
        n = sum((k + m) * size for _, k, m, size in _geometry(case))
    return {"bytes": float(n), "flops": 0.0}


def exact(case, seed):
    """Every output is bytes, equal or not."""
    return None
