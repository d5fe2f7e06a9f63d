"""Device memory that a context keeps for its next calls, and gives back."""
import numpy as np
import pytest
import torch

import glc

pytestmark = pytest.mark.gpu


def test_temporaries_of_a_large_call_stay_for_the_next():
    """1.1 * 10^9 int64 values take 8.8 GB of temporaries: mapped by the first call, kept afterwards."""
    ctx = glc.Context(0)
    n = 1_100_000_000
    v = torch.arange(n, dtype=torch.int64, device="cuda:0")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        glc.compress_device(ctx, glc.I64, v.data_ptr(), n, glc.FIXED).free()
        ctx.sync()
        assert before - torch.cuda.mem_get_info()[0] > 8 * n
    del v
    torch.cuda.empty_cache()
    ctx.close()


def test_memory_kept_by_the_other_pool_is_given_back_before_out_of_memory():
    """Compressing 128M int64 values from the host leaves about 2 GB of temporaries in their pool.  With
    600 MB of the device left, the pre-unpacked residuals (1 GB, from the columns' pool) fit only when
    that pool gives its memory back."""
    ctx = glc.Context(0)
    n = 128 << 20
    v = np.arange(n, dtype=np.int64) * 3
    v[::5] += 1
    col = glc.compress_device(ctx, glc.I64, v.ctypes.data, n, glc.FIXED, host=True)
    ctx.sync()
    left = 600 << 20
    hog = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda:0")
    try:
        glc.preunpack(ctx, col)
        pos = np.arange(0, n, 1_000_003, dtype=np.int32)
        got = np.zeros(len(pos), np.int64)
        glc.random_access_into(ctx, col, pos.ctypes.data, len(pos), got.ctypes.data, source=glc.SRC_PREUNPACKED,
                               host_in=True, host_out=True)
        assert np.array_equal(got, v[pos])
    finally:
        del hog
        torch.cuda.empty_cache()
        col.free()
        ctx.close()


def _wide_blob(ctx, n):
    """A column whose fields are as wide as its values, about 8 n bytes."""
    v = np.random.default_rng(7).integers(-(2 ** 62), 2 ** 62, n, dtype=np.int64)
    col = glc.compress_device(ctx, glc.I64, v.ctypes.data, n, glc.FIXED, host=True)
    blob = glc.serialize_host(ctx, col)
    col.free()
    return v, blob


def test_freed_deserialized_columns_give_their_memory_back():
    """Eight columns of 200 MB opened together and freed: no more than 512 MB stays with the context."""
    ctx = glc.Context(0)
    _, blob = _wide_blob(ctx, 25_000_000)
    cols = [glc.deserialize_host(ctx, glc.I64, blob) for _ in range(8)]
    ctx.sync()
    before = torch.cuda.mem_get_info()[0]
    for c in cols:
        c.free()
    ctx.sync()
    assert torch.cuda.mem_get_info()[0] - before > 8 * len(blob) - (544 << 20)
    ctx.close()


@pytest.mark.parametrize("n", [33_000_000, 34_000_000])
def test_deserialized_columns_on_both_sides_of_the_pool_limit(n):
    """A blob of 264 MB (from the pool) and one of 272 MB (its own allocations): opened twice, decoded and freed."""
    ctx = glc.Context(0)
    v, blob = _wide_blob(ctx, n)
    assert (len(blob) <= 256 << 20) == (n == 33_000_000)
    out = torch.zeros(n, dtype=torch.int64, device="cuda:0")
    for _ in range(2):
        col = glc.deserialize_host(ctx, glc.I64, blob)
        out.zero_()
        torch.cuda.synchronize()
        glc.decompress_into(ctx, col, out.data_ptr())
        ctx.sync()
        assert np.array_equal(out.cpu().numpy(), v)
        col.free()
    ctx.close()
