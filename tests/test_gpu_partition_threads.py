"""Variable compress from several host threads at once, each with a context and stream of its own: the merge
rounds are a launch whose CTAs wait for one another, and several such launches run side by side."""
import threading

import numpy as np
import pytest

import glc
from glc import workloads as W

pytestmark = pytest.mark.gpu


def test_variable_compress_from_three_threads(oracle):
    work = [W.piecewise_linear(1_500_000, seed=5, mean_segment=4_000), W.timestamps(900_011, seed=6),
            W.plain_small(400_003, seed=7)]
    wanted = [oracle.serialize(oracle.compress(v, "variable")) for v in work]
    ctxs = [glc.Context(0) for _ in work]
    failed = []

    def body(ctx, v, blob):
        try:
            for _ in range(15):
                col = glc.compress_device(ctx, glc.DTYPE_OF[v.dtype], v.ctypes.data, len(v), glc.VARIABLE, host=True)
                if glc.serialize_host(ctx, col) != blob:
                    failed.append("blob differs")
                col.free()
        except Exception as ex:  # reported to the test's thread
            failed.append(repr(ex))

    threads = [threading.Thread(target=body, args=a) for a in zip(ctxs, work, wanted)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for ctx in ctxs:
        ctx.close()
