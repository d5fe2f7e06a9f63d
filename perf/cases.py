"""The calls whose time matters to a user of this library, over the sizes, element types and options
they are made with.

A case is one of these tasks, each a pass through the library's public calls (the Python binding,
or the C entry where the binding has no wrapper), on data that already lies where such a program
has it:

* ``compress``  a column in device memory is compressed (fixed partitions, the model-cost
                partitioner, or the reference's GPU partitioner) and its blob written to a device
                buffer; the column of the pass before is freed first.
* ``decode``    a resident column is decoded in full into a device buffer.
* ``lookup``    values at a device array of positions are read from a resident column.
* ``batch``     many columns of mixed element types are compressed and decoded together.
* ``reload``    a blob in host memory (as read from a file) is deserialized, the column decoded on
                the device, and the column freed.
* ``serve``     a burst of lookup and range requests is submitted to a server of resident columns
                and waited for.

Columns (``data``): ``piecewise`` = straight segments of about 50,000 values with jumps, slopes and
noise widths that differ per segment; ``timestamps`` = cumulative sums of exponential gaps;
``linear`` = one line and noise of a drawn width.  The model-cost partitioner is what the
reference's users get by default for variable partitions, so it is measured at three sizes.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "g-leco_b200"))
import glc  # noqa: E402

CODE = {"i32": glc.I32, "i64": glc.I64, "u64": glc.U64, "u32": glc.U32}
SIZE = {"i32": 4, "i64": 8, "u64": 8, "u32": 4}
WORD = {"i32": torch.int32, "i64": torch.int64, "u64": torch.int64, "u32": torch.int32}  # bit patterns
MODE = {"fixed": glc.FIXED, "variable": glc.VARIABLE, "v6": glc.VARIABLE_V6}
MOST = 200_000_000  # values of the longest column (the published datasets' size)


def listed():
    return [
        # a whole analytics column scanned: the size of the published datasets, model-cost partitions
        dict(name="decode_var_u64_200M", task="decode", dtype="u64", data="piecewise", n=MOST, mode="variable", length=0),
        # a small resident column scanned: launch latency counts
        dict(name="decode_fix1024_i32_1M", task="decode", dtype="i32", data="linear", n=1 << 20, mode="fixed", length=1024),
        # a join or index probe: more positions than values, half uniform and half hot partitions
        dict(name="lookup_fix_i64_64M_100M", task="lookup", dtype="i64", data="timestamps", n=64_000_000, mode="fixed",
             length=4096, count=100_000_000),
        # a query's row fetch: a few thousand positions of a column with model-cost partitions
        dict(name="lookup_var_u64_5M_10k", task="lookup", dtype="u64", data="piecewise", n=5_000_003, mode="variable",
             length=0, count=10_007),
        # bulk ingest at the default fixed partition length
        dict(name="compress_fix4096_u64_200M", task="compress", dtype="u64", data="piecewise", n=MOST, mode="fixed", length=4096),
        # ingest of one small column chunk
        dict(name="compress_fix1024_i32_1M", task="compress", dtype="i32", data="linear", n=1 << 20, mode="fixed", length=1024),
        # bulk ingest with the best compression
        dict(name="compress_var_u64_200M", task="compress", dtype="u64", data="piecewise", n=MOST, mode="variable", length=0),
        # an ordinary column, of odd length, with the best compression
        dict(name="compress_var_i64_3M", task="compress", dtype="i64", data="timestamps", n=3_000_017, mode="variable", length=0),
        # sorted 32-bit keys with the reference's GPU partitioner
        dict(name="compress_v6_u32_30M", task="compress", dtype="u32", data="timestamps", n=30_000_001, mode="v6", length=0),
        # a table's columns, or one window of a stream, compressed and read back together
        dict(name="batch_1024", task="batch", columns=1024, median=100_000, length=0),
        # a stored column opened and read
        dict(name="reload_var_u64_2M", task="reload", dtype="u64", data="piecewise", n=2_000_003, mode="variable", length=0),
        # a burst of requests against resident columns
        dict(name="serve_256", task="serve", n=20_000_000, columns=6, requests=256, lookups=0.8, longest=65_536),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def _drawn_column(rng, lo, hi):
    dtype = rng.choice(["u64", "u64", "i64", "i64", "u32", "i32"])
    data = rng.choice(["piecewise", "timestamps", "linear"] if SIZE[dtype] == 8 else ["timestamps", "linear"])
    mode = rng.choice(["fixed", "fixed", "variable", "variable", "v6"])
    length = rng.choice([512, 1000, 1024, 2048, 4096, 4096]) if mode == "fixed" else 0
    return dict(dtype=dtype, data=data, n=_log(rng, lo, hi), mode=mode, length=length)


def draw(rng):
    task = rng.choice(["compress", "compress", "compress", "decode", "decode", "lookup", "batch", "reload", "serve"])
    if task == "compress":
        return dict(task=task, **_drawn_column(rng, 10_000, MOST))
    if task == "decode":
        return dict(task=task, source=rng.choice(["packed", "packed", "plain"]), **_drawn_column(rng, 200_000, MOST))
    if task == "lookup":
        return dict(task=task, source=rng.choice(["packed", "packed", "plain"]), count=_log(rng, 10_000, 50_000_000),
                    **_drawn_column(rng, 1_000_000, 64_000_000))
    if task == "batch":
        return dict(task=task, columns=_log(rng, 8, 1024), median=_log(rng, 5_000, 100_000),
                    length=rng.choice([0, 0, 1024, 4096]))
    if task == "reload":
        return dict(task=task, **_drawn_column(rng, 10_000, 8_000_000))
    return dict(task=task, n=_log(rng, 100_000, 20_000_000), columns=rng.randint(1, 6), requests=_log(rng, 1, 1024),
                lookups=rng.choice([0.5, 0.8, 1.0]), longest=_log(rng, 100, 65_536))


# ---- data ----------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _piecewise(n, g, dtype):
    """Segments of Poisson(50,000) values, slope U{1..10^6}, jump U{0..2^40}, noise U[0, 2^b) with b of
    {0, 4, 8, 16, 24}; below 2^53 throughout."""
    at_most = n // 50_000 * 2 + 64
    lens = torch.poisson(torch.full((at_most,), 50_000.0, device="cuda"), generator=g).clamp_min(1).to(torch.int64)
    ends = torch.cumsum(lens, 0)
    s = int(torch.searchsorted(ends, torch.tensor([n], device="cuda")).item()) + 1
    lens = lens[:s].clone()
    lens[-1] -= int(ends[s - 1].item()) - n
    starts = torch.cumsum(lens, 0) - lens
    slope = torch.randint(1, 1_000_001, (s,), device="cuda", generator=g)
    jump = torch.randint(0, (1 << 40) + 1, (s,), device="cuda", generator=g)
    bits = torch.tensor([0, 4, 8, 16, 24], device="cuda")[torch.randint(0, 5, (s,), device="cuda", generator=g)]
    span = slope * (lens - 1)
    base = torch.cumsum(jump, 0) + torch.cumsum(span, 0) - span
    seg = torch.repeat_interleave(torch.arange(s, device="cuda"), lens, output_size=n)
    v = torch.arange(n, device="cuda") - starts[seg]
    v *= slope[seg]
    v += base[seg]
    noise = torch.randint(0, 1 << 24, (n,), device="cuda", generator=g)
    noise &= ((torch.ones_like(bits) << bits) - 1)[seg]
    v += noise
    return v


def _timestamps(n, g, dtype):
    """Sums of exponential gaps of mean 1000, or less where the type would not hold them."""
    top = {"i32": 2.0e9, "u32": 4.1e9}.get(dtype, 1e18)
    gaps = torch.empty(n, device="cuda", dtype=torch.float64).exponential_(max(1e-3, n / top), generator=g)
    return torch.cumsum(torch.round(gaps).to(torch.int64), 0)


def _linear(n, g, dtype):
    """intercept + slope * i + noise: slope up to 10^4 (less where the type would not hold it), noise of
    a drawn width up to 20 bits."""
    a, slope, w = (int(x) for x in torch.randint(0, 1 << 30, (3,), device="cuda", generator=g).tolist())
    slope = min(slope % 10_001, (1 << 30) // n) if SIZE[dtype] == 4 else slope % 10_001
    v = torch.arange(n, device="cuda") * slope
    v += a % (1 << 20)
    v += torch.randint(0, 1 << (w % 21), (n,), device="cuda", generator=g)
    return v


DATA = {"piecewise": _piecewise, "timestamps": _timestamps, "linear": _linear}


def _values(data, dtype, n, seed):
    return DATA[data](n, _generator(seed), dtype).to(WORD[dtype])


def _positions(n, count, seed):
    """Half of the positions uniform, half in partitions of 4096 drawn by Zipf(1.1)."""
    g = _generator(seed + 1)
    parts = (n + 4095) // 4096
    half = count // 2
    uniform = torch.randint(0, n, (count - half,), device="cuda", generator=g, dtype=torch.int32)
    weight = torch.arange(1, parts + 1, device="cuda", dtype=torch.float64) ** -1.1
    edge = torch.cumsum(weight / weight.sum(), 0)
    rank = torch.searchsorted(edge, torch.rand(half, device="cuda", generator=g, dtype=torch.float64)).clamp_max(parts - 1)
    at = torch.randperm(parts, device="cuda", generator=g)[rank] * 4096
    at += torch.randint(0, 4096, (half,), device="cuda", generator=g)
    return torch.cat([uniform, at.clamp_max(n - 1).to(torch.int32)])


def _batch_specs(case, seed):
    """Lengths log-normal about the median, in [1024, 40 medians]; element types mixed.  Lengths and types are
    the table's (the same for every seed), the lines the seed's."""
    k = case["columns"]
    rng = np.random.default_rng(k)
    lens = np.clip(rng.lognormal(math.log(case["median"]), 1.0, k), 1024, 40 * case["median"]).astype(np.int64)
    lens = np.maximum(1024, (lens * (case["median"] * 1.65 * k / lens.sum())).astype(np.int64))
    wide = rng.integers(0, 3, k)  # 0: i32, 1: i64, 2: u64
    rng = np.random.default_rng(seed)
    slope = rng.integers(0, 10_001, k)
    slope = np.where(wide == 0, np.minimum(slope, (1 << 30) // lens), slope)
    return lens, wide, slope, rng.integers(0, 1 << 20, k), rng.integers(0, 21, k)


def _batch_values(case, seed):
    """The columns' values back to back, each from a 16-byte boundary: (4-byte words, 8-byte words, and for
    each column its type, length and first word)."""
    lens, wide, slope, a, w = _batch_specs(case, seed)
    g = _generator(seed)
    flats, first = [], np.zeros(len(lens), np.int64)
    for narrow in (True, False):
        ids = np.flatnonzero((wide == 0) == narrow)
        room = (lens[ids] + 3) // 4 * 4
        first[ids] = np.cumsum(room) - room
        total = max(4, int(room.sum()))
        if len(ids):
            d = [torch.from_numpy(x[ids]).cuda() for x in (first, slope, a, w)]
            col = torch.repeat_interleave(torch.arange(len(ids), device="cuda"), torch.from_numpy(room).cuda(), output_size=total)
            v = (torch.arange(total, device="cuda") - d[0][col]) * d[1][col] + d[2][col]
            noise = torch.randint(0, 1 << 20, (total,), device="cuda", generator=g)
            v += noise & ((torch.ones_like(d[3]) << d[3]) - 1)[col]
        else:
            v = torch.zeros(total, device="cuda", dtype=torch.int64)
        flats.append(v.to(torch.int32) if narrow else v)
    return flats[0], flats[1], lens, wide, first


# ---- cases ---------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    return glc.Context(0)


def _compress(case, v):
    return glc.compress_device(_context(), CODE[case["dtype"]], v.data_ptr(), v.numel(), MODE[case["mode"]], fixed_len=case["length"] or 4096)


def _serve_columns(case, seed):
    kinds = [("u64", "piecewise", "variable"), ("i64", "timestamps", "fixed"), ("i64", "linear", "fixed")]
    for k in range(case["columns"]):
        dtype, data, mode = kinds[k % 3]
        yield dict(dtype=dtype, mode=mode, length=0), _values(data, dtype, case["n"], seed * 16 + k)


def _serve_requests(case, seed):
    """Columns at random; lookup counts and range lengths spread over their logarithm (the same mix for every
    seed: it is the load; columns, ranges and positions are the seed's)."""
    k = case["requests"]
    rng = np.random.default_rng(k)
    look = rng.random(k) < case["lookups"]
    count = np.exp(rng.uniform(0, math.log(case["longest"]), k)).astype(np.int64).clip(1, case["n"])
    rng = np.random.default_rng(seed)
    column = rng.integers(0, case["columns"], k)
    first = np.where(look, 0, (rng.random(k) * (case["n"] - count + 1)).astype(np.int64))
    # a range's output lies as its values do in a whole decode: (out - first) a multiple of 16 bytes
    room = (count + 3) // 2 * 2
    at = np.cumsum(room) - room + first % 2
    return look, column, count, first, at, int(room.sum())


def prepare(case, seed):
    ctx, task = _context(), case["task"]
    st = {"case": case, "ctx": ctx}
    if task in ("compress", "decode", "lookup", "reload"):
        v = _values(case["data"], case["dtype"], case["n"], seed)
        torch.cuda.synchronize()  # the library works on the context's own stream
    if task == "compress":
        st["values"] = v
        st["blob"] = torch.zeros(v.numel() * v.element_size() * 9 // 8 + 64 * (v.numel() // 128 + 64), dtype=torch.uint8, device="cuda")
        st["col"] = None
    elif task in ("decode", "lookup"):
        st["col"] = _compress(case, v)
        st["source"] = glc.SRC_PACKED
        if case.get("source") == "plain":
            glc.preunpack(ctx, st["col"])
            st["source"] = glc.SRC_PREUNPACKED
        if task == "lookup":
            st["pos"] = _positions(case["n"], case["count"], seed)
        st["out"] = torch.empty(case["n"] if task == "decode" else case["count"], dtype=WORD[case["dtype"]], device="cuda")
    elif task == "reload":
        col = _compress(case, v)
        st["blob"] = glc.serialize_host(ctx, col)
        col.free()
        st["out"] = torch.empty(case["n"], dtype=WORD[case["dtype"]], device="cuda")
    elif task == "batch":
        st["narrow"], st["broad"], lens, wide, first = _batch_values(case, seed)
        st["outs"] = torch.empty_like(st["narrow"]), torch.empty_like(st["broad"])
        for f, o in zip((st["narrow"], st["broad"]), st["outs"]):
            o.copy_(f)  # the room between columns keeps its words
        st["dtypes"] = np.array([glc.I32, glc.I64, glc.U64], np.int32)[wide]
        st["ns"] = lens
        st["in_ptrs"] = np.where(wide == 0, st["narrow"].data_ptr() + 4 * first, st["broad"].data_ptr() + 8 * first).astype(np.uint64)
        st["out_ptrs"] = np.where(wide == 0, st["outs"][0].data_ptr() + 4 * first, st["outs"][1].data_ptr() + 8 * first).astype(np.uint64)
        st["batch"] = None
    else:
        cols = []
        for spec, v in _serve_columns(case, seed):
            torch.cuda.synchronize()
            cols.append(_compress(spec, v))
            del v
        ctx.sync()
        st["server"] = glc.Server(ctx, budget_bytes=8 << 30)
        ids = np.array([st["server"].admit(c) for c in cols], np.int32)
        look, column, count, first, at, total = _serve_requests(case, seed)
        st["out"] = torch.zeros(total, dtype=torch.int64, device="cuda")
        where = np.where(look, np.cumsum(np.where(look, count, 0)) - np.where(look, count, 0), 0)
        st["pos"] = _positions(case["n"], max(1, int(count[look].sum())), seed)
        r = st["requests"] = glc.requests(case["requests"])
        r["kind"] = np.where(look, glc.REQ_LOOKUP, glc.REQ_RANGE)
        r["column"], r["first"], r["count"], r["tag"] = ids[column], first, count, np.arange(len(r))
        r["positions"] = np.where(look, st["pos"].data_ptr() + 4 * where, 0)
        r["out"] = st["out"].data_ptr() + 8 * at
    torch.cuda.synchronize()
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    task = case["task"]
    if task == "compress":
        if st["col"] is not None:
            st["col"].free()
        st["col"] = col = _compress(case, st["values"])
        size = ctypes.c_uint64()
        ctx.check(ctx.lib.glc_serialize(ctx.handle, col.handle, st["blob"].data_ptr(), st["blob"].numel(), 0, 0, ctypes.byref(size), None))
        return {"blob": st["blob"], "size": size.value}  # the blob, and zeros after it
    if task == "decode":
        glc.decompress_into(ctx, st["col"], st["out"].data_ptr(), source=st["source"])
        return st["out"]
    if task == "lookup":
        glc.random_access_into(ctx, st["col"], st["pos"].data_ptr(), case["count"], st["out"].data_ptr(), source=st["source"])
        return st["out"]
    if task == "reload":
        col = glc.deserialize_host(ctx, CODE[case["dtype"]], st["blob"])
        glc.decompress_into(ctx, col, st["out"].data_ptr())
        col.free()
        return st["out"]
    if task == "batch":
        if st["batch"] is not None:
            st["batch"].free()
        st["batch"] = b = glc.Batch.compress(ctx, st["dtypes"], st["in_ptrs"], st["ns"], fixed_len=case["length"])
        b.decompress(st["out_ptrs"])
        return {"narrow": st["outs"][0], "broad": st["outs"][1], "size": b.compressed_size}
    st["server"].submit(st["requests"])
    st["server"].drain()
    st["server"].poll(case["requests"])
    return st["out"]


def exact(case, seed):
    task = case["task"]
    if task in ("decode", "reload"):
        return _values(case["data"], case["dtype"], case["n"], seed)
    if task == "lookup":
        return _values(case["data"], case["dtype"], case["n"], seed)[_positions(case["n"], case["count"], seed).long()]
    if task == "batch":
        narrow, broad = _batch_values(case, seed)[:2]
        return {"narrow": narrow, "broad": broad, "size": None}
    if task == "serve":
        look, column, count, first, at, total = _serve_requests(case, seed)
        out, pos, used = torch.zeros(total, dtype=torch.int64, device="cuda"), _positions(case["n"], max(1, int(count[look].sum())), seed).long(), 0
        cols = [v for _, v in _serve_columns(case, seed)]
        for k in range(len(look)):
            v, c = cols[column[k]], int(count[k])
            out[at[k]: at[k] + c] = v[pos[used: used + c]] if look[k] else v[first[k]: first[k] + c]
            used += c if look[k] else 0
        return out
    return None  # a blob's bytes are the format's, not computed numbers


def _field_bits(case):
    """Bits a value takes in the compressed column, about."""
    if case["data"] == "timestamps":
        return min(17.0, 7.0 + math.log2(max(1.0, 4e9 / case["n"]))) if SIZE[case["dtype"]] == 4 else 17.0
    return 12.9 if case["data"] == "piecewise" else 11.0


def work(case):
    task = case["task"]
    if task == "serve":
        # the mean of exp(U(0, log m)) is (m - 1) / log m; a lookup reads a position and a field
        values = case["requests"] * (case["longest"] - 1) / math.log(case["longest"])
        return {"bytes": values * (8 + case["lookups"] * 8 + (1 - case["lookups"]) * 1.7)}
    if task == "batch":  # in and out, and the compressed columns written and read
        values = case["columns"] * case["median"] * 1.65
        return {"bytes": values * 2 * (20 / 3 + 11 / 8)}
    raw, packed = case["n"] * SIZE[case["dtype"]], case["n"] * _field_bits(case) / 8
    if task == "lookup":  # positions and values, and the sectors of the fields, each at most once
        q = case["count"]
        fields = case["n"] * 8 if case.get("source") == "plain" else packed
        return {"bytes": q * (4 + SIZE[case["dtype"]]) + min(32 * q, fields)}
    if task == "decode" and case.get("source") == "plain":
        return {"bytes": raw + 8 * case["n"]}
    if task == "reload":  # the blob crosses to the device, is read there, and the values written
        return {"bytes": raw + 2 * packed}
    return {"bytes": raw + packed}
