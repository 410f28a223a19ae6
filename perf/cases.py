"""What the performance of this library is measured on: calls as a program
that converts layouts makes them, through the Python binding, over the sizes,
element widths and operations of the benchmark's workloads (bench.py).

Every conversion is in place, so a pass converts the state's own buffer and
returns it.  Buffers hold random bits; elements are moved and never computed
with, so they are integer tensors of the element's width.
"""
import math

import torch

from libmarshal_gb300 import lm

DTYPES = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}

# op -> the dimensions a case of it names
DIMS = {
    "transpose": ("M", "N"),          # [M][N] -> [N][M], any M and N
    "staged": ("A", "a", "B", "b"),   # the same, given as [A*a][B*b]
    "stack": ("T", "M", "N"),         # T matrices, each transposed
    "aos_asta": ("h", "w", "t"),      # [h][w] -> [h/t][w][t]
    "asta_aos": ("h", "w", "t"),      # and back
    "soa_asta": ("h", "w", "t"),      # [w][h] -> [h/t][w][t]
    "asta_soa": ("h", "w", "t"),      # and back
    "padding": ("x", "y", "pad"),     # [y][x] -> [y][pad]
    "unpadding": ("x", "y", "pad"),   # and back, zeros behind the rows
    "batch": ("jobs", "jobs_seed"),   # a list of mixed conversions
}


def listed():
    return [
        # A handful of small matrices or records at a time: what one call
        # costs, whatever it moves.
        {"name": "transpose_48x64_f32", "op": "transpose", "e": 4,
         "M": 48, "N": 64},
        # 65,536 structs of seven floats to the tiled layout, the
        # reference's own small AoS -> ASTA workload; stays in L2.
        {"name": "aos_asta_65536x7_f32", "op": "aos_asta", "e": 4,
         "h": 65536, "w": 7, "t": 32},
        # An odd byte image: neither side is a multiple of anything.
        {"name": "transpose_3301x2503_u8", "op": "transpose", "e": 1,
         "M": 3301, "N": 2503},
        # The rectangular matrix of the reference's staged transposition,
        # with the tile factors that its planner takes.
        {"name": "staged_7200x1800_f32", "op": "staged", "e": 4,
         "A": 72, "a": 100, "B": 18, "b": 100},
        # A square matrix, 268 MB, as linear algebra transposes it.
        {"name": "transpose_8192x8192_f32", "op": "transpose", "e": 4,
         "M": 8192, "N": 8192},
        # The headline: coprime sides, 805 MB.
        {"name": "transpose_16384x12289_f32", "op": "transpose", "e": 4,
         "M": 16384, "N": 12289},
        # The largest: 4.2 GB of doubles.
        {"name": "transpose_32768x16000_f64", "op": "transpose", "e": 8,
         "M": 32768, "N": 16000},
        # Field arrays to the tiled layout: 24 float fields, 32 records to
        # a tile, a record count that is no power of two.
        {"name": "soa_asta_6000000x24_f32", "op": "soa_asta", "e": 4,
         "h": 6000000, "w": 24, "t": 32},
        # Tiles of sixteen half-precision records back to field arrays:
        # units of one sector.
        {"name": "asta_soa_2000000x101_f16", "op": "asta_soa", "e": 2,
         "h": 2000000, "w": 101, "t": 16},
        # Tiles back to structs, wide ones: 500 halves each, a tile of 64 KB.
        {"name": "asta_aos_262144x500_f16", "op": "asta_aos", "e": 2,
         "h": 262144, "w": 500, "t": 64},
        # Rows padded to whole 128-byte lines before a kernel that wants
        # them so (and the first step of the reference's general flow).
        {"name": "padding_8192x12289_f32", "op": "padding", "e": 4,
         "x": 12289, "y": 8192, "pad": 12320},
        # Many uneven matrices of all widths in one call.
        {"name": "batch_512_mixed", "op": "batch", "e": 0,
         "jobs": 512, "jobs_seed": 1},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    op = rng.choice(["transpose", "transpose", "staged", "stack", "aos_asta",
                     "asta_aos", "soa_asta", "asta_soa", "padding",
                     "unpadding", "batch"])
    e = rng.choice([1, 2, 4, 8])
    if op == "batch":
        return {"op": op, "e": 0, "jobs": _log_uniform(rng, 16, 512),
                "jobs_seed": rng.randrange(1, 1 << 20)}
    # payload from 12 KB to 1 GB
    n = max(256, _log_uniform(rng, 12 << 10, 1 << 30) // e)
    if op in ("transpose", "padding", "unpadding"):
        if op == "transpose" and rng.random() < 0.25:
            m = max(16, math.isqrt(n))
            return {"op": op, "e": e, "M": m, "N": m}
        m = _log_uniform(rng, 16, max(16, n // 16))
        k = max(16, n // m)
        if op == "transpose":
            return {"op": op, "e": e, "M": m, "N": k}
        y, x = max(16, m // 2), k
        # rows rounded up to whole units
        unit = rng.choice([u for u in (16, 32, 128) if u <= x])
        return {"op": op, "e": e, "x": x, "y": y,
                "pad": (x // unit + 1) * unit}
    if op == "staged":
        a, b = rng.randint(24, 100), rng.randint(24, 100)
        rest = max(4, n // (a * b))
        A = _log_uniform(rng, 2, max(2, rest // 2))
        return {"op": op, "e": e, "A": A, "a": a,
                "B": max(2, rest // A), "b": b}
    if op == "stack":
        T = _log_uniform(rng, 2, 256)
        m = _log_uniform(rng, 8, max(8, n // T // 8))
        return {"op": op, "e": e, "T": T, "M": m, "N": max(8, n // T // m)}
    t = rng.choice([16, 32, 64])
    w = _log_uniform(rng, 2, 1024)
    return {"op": op, "e": e, "h": max(2, n // (w * t)) * t, "w": w, "t": t}


def _elements(case):
    d = [case[k] for k in DIMS[case["op"]]]
    if case["op"] in ("padding", "unpadding"):
        return case["y"] * case["pad"]
    if case["op"] in ("aos_asta", "asta_aos", "soa_asta", "asta_soa"):
        return case["h"] * case["w"]
    return math.prod(d)


def _batch_jobs(case):
    """(op, dims, element bytes, byte offset) of each job: sides
    log-uniform in [16, 4096], widths uniform, half of them AoS -> ASTA with
    tiles of 16, 32 or 64 and half transpositions; and the bytes in all."""
    import random
    rng = random.Random(case["jobs_seed"])
    jobs, off = [], 0
    for _ in range(case["jobs"]):
        h, w = _log_uniform(rng, 16, 4096), _log_uniform(rng, 16, 4096)
        e = rng.choice([1, 2, 4, 8])
        if rng.random() < 0.5:
            t = rng.choice([16, 32, 64])
            h = -(-h // t) * t
            jobs.append(("aos_asta", (h, w, t), e, off))
        else:
            jobs.append(("transpose", (h, w), e, off))
        off += -(-h * w * e // 256) * 256
    return jobs, off


def _random(elements, e, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    info = torch.iinfo(DTYPES[e])
    buf = torch.empty(elements, dtype=DTYPES[e], device="cuda")
    return buf.random_(info.min, info.max, generator=g)


def prepare(case, seed):
    if case["op"] == "batch":
        jobs, size = _batch_jobs(case)
        buf = _random(size // 8, 8, seed)
        base = buf.data_ptr()
        code = {"aos_asta": lm.OP_AOS_ASTA, "transpose": lm.OP_TRANSPOSE}
        return {"case": case, "buf": buf, "batch": lm.Batch(),
                "jobs": [lm.job(base + off, code[op], dims, e)
                         for op, dims, e, off in jobs]}
    return {"case": case, "buf": _random(_elements(case), case["e"], seed)}


def run(state):
    case, buf = state["case"], state["buf"]
    op = case["op"]
    if op == "batch":
        state["batch"].run(state["jobs"])
        return buf
    d = [case[k] for k in DIMS[op]]
    if op == "transpose":
        lm.full_transpose(buf, d[0], d[1])
    elif op == "staged":
        lm.transpose(buf, *d)
    elif op == "stack":
        lm.transpose_0100(buf, d[0], d[1], d[2], 1)
    elif op == "padding":
        lm.padding(buf, d[0], d[1], d[2])
    elif op == "unpadding":
        lm.unpadding(buf, d[0], d[1], d[2])
    else:
        h, w, t = d
        if op == "aos_asta":
            lm.aos_asta(buf, h, w, t)
        elif op == "asta_aos":
            lm.transpose_0100(buf, h // t, w, t, 1)
        elif op == "soa_asta":
            lm.transpose_100(buf, w, h // t, t)
        else:
            lm.transpose_100(buf, h // t, w, t)
    return buf


def work(case):
    """Every element is read once and written once (padding writes its new
    columns and unpadding its zeros too; padding columns are not read)."""
    if case["op"] == "batch":
        return {"bytes": sum(2 * d[0] * d[1] * e for _, d, e, _ in _batch_jobs(case)[0]),
                "flops": 0}
    if case["op"] in ("padding", "unpadding"):
        return {"bytes": case["y"] * (case["x"] + case["pad"]) * case["e"],
                "flops": 0}
    return {"bytes": 2 * _elements(case) * case["e"], "flops": 0}


def _converted(op, d, src):
    """The conversion of the flat tensor `src`, out of place, by plain torch."""
    if op == "transpose":
        return src.view(d[0], d[1]).t().reshape(-1)
    if op == "staged":
        return src.view(d[0] * d[1], d[2] * d[3]).t().reshape(-1)
    if op == "stack":
        return src.view(d[0], d[1], d[2]).transpose(1, 2).reshape(-1)
    if op in ("padding", "unpadding"):
        x, y, pad = d
        out = torch.zeros_like(src)
        if op == "padding":
            out.view(y, pad)[:, :x] = src[:y * x].view(y, x)
        else:
            out[:y * x].view(y, x)[:] = src.view(y, pad)[:, :x]
        return out
    h, w, t = d
    if op == "aos_asta":
        return src.view(h // t, t, w).transpose(1, 2).reshape(-1)
    if op == "asta_aos":
        return src.view(h // t, w, t).transpose(1, 2).reshape(-1)
    if op == "soa_asta":
        return src.view(w, h // t, t).transpose(0, 1).reshape(-1)
    return src.view(h // t, w, t).transpose(0, 1).reshape(-1)


def exact(case, seed):
    if case["op"] == "batch":
        jobs, size = _batch_jobs(case)
        out = _random(size // 8, 8, seed)
        raw = out.view(torch.uint8)
        for op, dims, e, off in jobs:
            part = raw[off:off + dims[0] * dims[1] * e].view(DTYPES[e])
            part.copy_(_converted(op, dims, part))
        return out
    src = _random(_elements(case), case["e"], seed)
    return _converted(case["op"], [case[k] for k in DIMS[case["op"]]], src)
