"""Host-memory entry points around the size from which their copies are staged
by several threads, once a context has copied enough for them: arrays below
it, of whole pieces, with a short last piece, with more pieces than buffers,
and two contexts copying at once, each against the same call on device memory,
bit for bit."""
import os
import threading
from contextlib import closing, suppress
from pathlib import Path

import numpy as np
import pytest
import torch

from nimbus_b200 import cuda
from nimbus_b200.initial import Case, cloudy_state

pytestmark = pytest.mark.gpu
FIELDS = ("theta", "qv", "qc", "qr")


def _same(got, want, what):
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), what


def _cloudy(shape, seed):
    st, _ = cloudy_state(Case(*shape, 900.0, 850.0, 300.0, 4.0, seed=seed), seed=seed)
    return {k: st[k] for k in FIELDS + ("p", "rho")}


def _on_device(ctx, st):
    dev = {k: torch.from_numpy(v).cuda() for k, v in st.items()}
    torch.cuda.synchronize()
    ctx.check(ctx.kessler_step(cuda.kessler_args(dev, 300.0, 4.0, memory=cuda.MEMORY_DEVICE)))
    ctx.synchronize()
    return {k: dev[k].cpu().numpy() for k in FIELDS}


def _copier_threads():
    """Threads of this process that bear the copier's name."""
    found = 0
    for comm in Path("/proc/self/task").glob("*/comm"):
        with suppress(OSError):  # a thread that has just ended
            found += comm.read_text().strip() == "nimbus-copy"
    return found


def _warmed(ctx):
    """Copies host arrays until the device's copier is set up (64 MiB the
    ordinary way, then a call that starts its threads) and says whether they
    run: three beside the caller, or as many as there are cores for."""
    st = _cloudy((96, 95, 61), 1)
    for _ in range(5):  # ten copies of 2.1 MiB a call
        ctx.check(ctx.kessler_step(cuda.kessler_args({k: v.copy() for k, v in st.items()}, 300.0, 4.0)))
    return _copier_threads() == min(4, os.cpu_count()) - 1


# 2^18 floats are four pieces, the smallest array that is staged so; the next
# has a last piece of 8,880 bytes, the last more pieces than there are buffers.
@pytest.mark.parametrize("shape", [(64, 64, 63), (64, 64, 64), (43, 53, 116), (96, 95, 61)],
                         ids=["below", "pieces", "tail", "more"])
def test_host_arrays_give_the_device_result(shape):
    with closing(cuda.Context(0)) as ctx:
        assert _warmed(ctx)
        st = _cloudy(shape, 5)
        want = _on_device(ctx, st)
        for _ in range(3):
            got = {k: v.copy() for k, v in st.items()}
            ctx.check(ctx.kessler_step(cuda.kessler_args(got, 300.0, 4.0)))
            for k in FIELDS:
                _same(got[k], want[k], k)


def test_two_contexts_copy_at_once():
    """Both hold the device's copier, and the one that finds it busy copies the
    ordinary way."""
    shape = (96, 95, 61)
    states = [_cloudy(shape, 7 + t) for t in range(2)]
    with closing(cuda.Context(0)) as ctx:
        want = [_on_device(ctx, st) for st in states]
    got = [None, None]
    together = threading.Barrier(2)
    with closing(cuda.Context(0)) as holder:
        assert _warmed(holder)

        def work(t):
            with closing(cuda.Context(0)) as ctx:
                together.wait(60)
                for _ in range(8):
                    mine = {k: v.copy() for k, v in states[t].items()}
                    ctx.check(ctx.kessler_step(cuda.kessler_args(mine, 300.0, 4.0)))
                got[t] = mine

        threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(60)
    for t in range(2):
        for k in FIELDS:
            _same(got[t][k], want[t][k], f"{t} {k}")
