"""Bit-exact blobs beside the limits at which a call changes its way.

* the merge rounds count a list of up to 16,384 partitions in every CTA, longer ones by per-CTA counts
  with one more barrier;
* up to 16,384 bit counts are scanned by one CTA, more by three launches; four counts are one access
  where both arrays are 32-byte aligned;
* a host blob's metadata goes up as one copy where it lies in one piece of aligned words, else array by
  array.
"""
import struct

import numpy as np
import pytest
import torch

import glc

pytestmark = pytest.mark.gpu


def _blob(ctx, v, mode, length=4096):
    col = glc.compress_device(ctx, glc.DTYPE_OF[v.dtype], v.ctypes.data, len(v), mode, fixed_len=length, host=True)
    blob = glc.serialize_host(ctx, col)
    col.free()
    return blob


def _short_lines(n, dtype, most, seed):
    """A new line every 128 to 128 `most` values, at a multiple of 128: jumps of every size, so that some
    neighbours are worth merging and others are not."""
    rng = np.random.default_rng(seed)
    lens = 128 * rng.integers(1, most + 1, n // 128 + 1)
    seg = np.repeat(np.arange(len(lens)), lens)[:n]
    at = np.arange(n) - (np.cumsum(lens) - lens)[seg]
    base = (2.0 ** rng.uniform(0, 28, len(lens))).astype(np.int64) * rng.choice([-1, 1], len(lens))
    v = base[seg] + at * rng.integers(-3, 4, len(lens))[seg] + rng.integers(0, 4, n)
    return v.astype(dtype) if np.dtype(dtype).kind == "i" else (v + (1 << 30)).astype(dtype)


@pytest.mark.parametrize("dtype,most", [(np.int64, 2), (np.uint32, 3), (np.int32, 4), (np.uint64, 5)])
def test_many_short_partitions_match_the_oracle(glc_ctx, oracle, dtype, most):
    """39,000 blocks of 128 values: lists that stay above the limit, and lists that fall below it as they merge."""
    v = _short_lines(5_000_011, dtype, most, seed=most)
    assert _blob(glc_ctx, v, glc.VARIABLE) == oracle.serialize(oracle.compress(v, "variable"))


@pytest.mark.parametrize("blocks", [16_383, 16_384, 16_385])
def test_partition_lists_beside_the_short_limit(glc_ctx, oracle, blocks):
    """Runs of 128 equal values, far apart: the split makes one partition of each."""
    rng = np.random.default_rng(blocks)
    v = np.repeat(rng.integers(-(1 << 40), 1 << 40, blocks), 128)
    ours = _blob(glc_ctx, v, glc.VARIABLE)
    assert struct.unpack_from("<I", ours, 12)[0] == blocks
    assert ours == oracle.serialize(oracle.compress(v, "variable"))


@pytest.mark.parametrize("length", [100, 128])
@pytest.mark.parametrize("parts", [16_383, 16_384, 16_385])
def test_bit_offset_scans_beside_the_one_launch_limit(glc_ctx, oracle, parts, length):
    v = np.random.default_rng(parts).integers(0, 1 << 12, (parts - 1) * length + 7).astype(np.int32)
    assert _blob(glc_ctx, v, glc.FIXED, length) == oracle.serialize(oracle.compress(v, "fixed", length))


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 6, 7, 8])
def test_bit_offset_scans_at_every_alignment(glc_ctx, oracle, tiles):
    v = np.random.default_rng(tiles).integers(0, 1 << 30, tiles * 4096 - 5).astype(np.uint64)
    assert _blob(glc_ctx, v, glc.FIXED) == oracle.serialize(oracle.compress(v, "fixed", 4096))


def _moved(blob, how):
    """The same column with its metadata arrays elsewhere in the blob (header: 4 words, 8 array offsets, 2
    sizes, type size, checksum by rotate-add over the header with the checksum 0)."""
    h = list(struct.unpack_from("<4I8Q2Q2I4I", blob))
    P, at, delta = h[3], h[4:11], blob[h[11]:]
    lens = [4 * P, 4 * P, 4 * P, 32 * P, 4 * P, 8 * P, 8 * P]
    arrays = [blob[a:a + n] for a, n in zip(at, lens)]
    out = bytearray(120)
    for k in reversed(range(7)) if how == "reversed" else range(7):
        out += bytes({"odd": 1, "halves": 2, "far": 4096, "near": 4}.get(how, 0))
        h[4 + k] = len(out)
        out += arrays[k]
    out += bytes(-len(out) % 8)
    h[11] = len(out)
    h[15] = 0
    c = 0
    for x in struct.pack("<4I8Q2Q2I4I", *h):
        c = (c + x) & 0xFFFFFFFF
        c = ((c << 1) | (c >> 31)) & 0xFFFFFFFF
    h[15] = c
    out[:120] = struct.pack("<4I8Q2Q2I4I", *h)
    return bytes(out + delta)


@pytest.mark.parametrize("how", ["packed", "near", "reversed", "halves", "odd", "far"])
@pytest.mark.parametrize("n", [1, 130, 200_003])
def test_blobs_with_moved_arrays_open_as_the_column_they_hold(glc_ctx, oracle, how, n):
    v = _short_lines(n, np.int64, 5, seed=n)
    blob = _blob(glc_ctx, v, glc.VARIABLE)
    col = glc.deserialize_host(glc_ctx, glc.I64, _moved(blob, how))
    assert col is not None
    assert glc.serialize_host(glc_ctx, col) == blob
    out = torch.zeros(n, dtype=torch.int64, device="cuda:0")
    torch.cuda.synchronize()
    glc.decompress_into(glc_ctx, col, out.data_ptr())
    glc_ctx.sync()
    assert np.array_equal(out.cpu().numpy(), v)
    col.free()
