"""Host-memory entry points around the size from which their copies are staged
by several threads: arrays below it, of whole pieces, with a last piece of a
few bytes, with more pieces than buffers, and two contexts copying at once,
each against the same call on device memory, bit for bit."""
import threading
from contextlib import closing

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


# 2^18 floats are four pieces, the smallest array that is staged so.
@pytest.mark.parametrize("shape", [(64, 64, 63), (64, 64, 64), (43, 53, 116), (96, 95, 61)],
                         ids=["below", "pieces", "tail", "more"])
def test_host_arrays_give_the_device_result(shape):
    with closing(cuda.Context(0)) as ctx:
        st = _cloudy(shape, 5)
        want = _on_device(ctx, st)
        for _ in range(5):  # the first ones go the ordinary way while the copier is set up
            got = {k: v.copy() for k, v in st.items()}
            ctx.check(ctx.kessler_step(cuda.kessler_args(got, 300.0, 4.0)))
            for k in FIELDS:
                _same(got[k], want[k], k)


def test_two_contexts_copy_at_once():
    shape = (96, 95, 61)
    states = [_cloudy(shape, 7 + t) for t in range(2)]
    with closing(cuda.Context(0)) as ctx:
        want = [_on_device(ctx, st) for st in states]
    got = [None, None]

    def work(t):
        with closing(cuda.Context(0)) as ctx:
            for _ in range(4):
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
