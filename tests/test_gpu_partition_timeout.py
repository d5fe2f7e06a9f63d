"""A run-out wait of the variable partitioner's merge rounds is a timeout, and the context stays usable.

With GLC_TEST_EXPIRE_FIRST_WAIT=2 when a context is created, the CTAs of that context's next merge
launch wait for one arrival more than there are, for a millisecond: every one of them gives up at the
first barrier and leaves.  The call must return GLC_ERR_TIMEOUT, and the next one on the same context
must give the oracle's blob.
"""
import numpy as np
import pytest

import glc
from glc import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["compress", "partition"])
def test_run_out_barrier_is_a_timeout_and_the_next_call_is_exact(monkeypatch, oracle, call):
    monkeypatch.setenv("GLC_TEST_EXPIRE_FIRST_WAIT", "2")
    ctx = glc.Context(0)
    monkeypatch.delenv("GLC_TEST_EXPIRE_FIRST_WAIT")
    v = W.piecewise_linear(300_000, seed=23, mean_segment=5_000)
    with pytest.raises(glc.GlcError) as err:
        if call == "compress":
            glc.compress_device(ctx, glc.U64, v.ctypes.data, len(v), glc.VARIABLE, host=True)
        else:
            glc.partition_variable(ctx, v)
    assert err.value.status == glc.ERR_TIMEOUT
    col = glc.compress_device(ctx, glc.U64, v.ctypes.data, len(v), glc.VARIABLE, host=True)
    assert glc.serialize_host(ctx, col) == oracle.serialize(oracle.compress(v, "variable"))
    col.free()
    ctx.close()
