"""Single members read, written and recorded from threads that have made no
CUDA call yet, or have another device current, with padded columns (every nz
modulo four) and without."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from nimbus_b200 import cuda
from nimbus_b200.initial import Case, perturbed_state
from nimbus_b200.run import EngineRun

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "rho", "p", "theta", "qv", "qc", "qr")


def _members(run, levels=(8, 9, 10, 11)):
    out = []
    for m, nz in enumerate(levels):
        case = Case(9, 8, nz, 900.0, 850.0, 600.0, 2.0, seed=2, member=m)
        st, base = perturbed_state(case, seed=60 + m)
        out.append((run.admit(case, st, base, n_substeps=2), st))
    return out


def _in_thread(work):
    failed = []

    def body():
        try:
            work()
        except BaseException as error:  # handed to the test's own thread
            failed.append(error)

    t = threading.Thread(target=body)
    t.start()
    t.join(120)
    assert not t.is_alive()
    if failed:
        raise failed[0]


def _read_and_write(run, members):
    for mid, st in members:
        got = run.read(mid)
        for k in FIELDS:
            assert np.array_equal(got[k].view(np.uint32), st[k].view(np.uint32)), k
        st["theta"] = st["theta"] + np.float32(1.0)
        run.engine.write(mid, st)
        got = run.read(mid)
        assert np.array_equal(got["theta"], st["theta"])


def test_members_move_in_a_new_thread():
    ctx = cuda.Context(0)
    run = EngineRun(ctx)
    members = _members(run)
    _in_thread(lambda: _read_and_write(run, members))
    run.close()
    ctx.close()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs a second device")
def test_members_move_with_another_device_current():
    ctx = cuda.Context(1)
    run = EngineRun(ctx)
    members = _members(run)

    def work():
        torch.cuda.set_device(0)
        torch.zeros(1, device="cuda:0")
        _read_and_write(run, members)

    _in_thread(work)
    run.close()
    ctx.close()


def _pool_high_water(reset=False):
    """Most bytes in use at once of the device's default memory pool since the
    last reset."""
    driver = ctypes.CDLL("libcuda.so.1")
    pool, value = ctypes.c_void_p(), ctypes.c_uint64(0)
    assert driver.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    used_high = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    if reset:
        assert driver.cuMemPoolSetAttribute(pool, used_high, ctypes.byref(value)) == 0
    assert driver.cuMemPoolGetAttribute(pool, used_high, ctypes.byref(value)) == 0
    return value.value


def test_a_member_moves_within_its_own_memory():
    """Admission, read, write and history of a padded member take no device
    memory beyond member_bytes: what fits at admission keeps fitting."""
    ctx = cuda.Context(0)
    run = EngineRun(ctx)
    first = _members(run, levels=(9,))
    _read_and_write(run, first)
    case = Case(41, 40, 13, 900.0, 850.0, 600.0, 2.0, seed=2)
    st, base = perturbed_state(case, seed=70)
    desc = cuda.member_desc(case.shape, (case.dx, case.dy, case.dz), case.dt, 2, case.bc, base)
    before = _pool_high_water(reset=True)
    mid = run.engine.admit(desc, st)
    run.engine.synchronize()
    assert _pool_high_water() - before <= run.engine.member_bytes(desc) + 4096  # the pool's granularity
    held = _pool_high_water(reset=True)
    _read_and_write(run, [(mid, st)])
    frame = np.empty(9 * st["u"].size, np.float32)
    run.engine.history_async(mid, cuda.HISTORY_CORE, frame)
    run.engine.synchronize()
    assert _pool_high_water() == held
    run.close()
    ctx.close()


@pytest.mark.parametrize("names", [("rho",), ("u",), ("w", "qr"), ("v", "theta", "qc")], ids="-".join)
def test_history_of_some_fields_of_a_padded_member(names):
    ctx = cuda.Context(0)
    run = EngineRun(ctx)
    for mid, st in _members(run, levels=(9, 10, 11)):
        want = np.empty(9 * st["u"].size, np.float32)
        run.engine.history_async(mid, cuda.HISTORY_CORE, want)
        got = np.full(len(names) * st["u"].size, np.nan, np.float32)
        run.engine.history_async(mid, cuda.history_mask(names), got)
        run.engine.synchronize()
        want, got = (x.reshape(-1, *st["u"].shape) for x in (want, got))
        for k, frame in zip(names, got):
            assert np.array_equal(frame.view(np.uint32), want[FIELDS.index(k)].view(np.uint32)), k
    run.close()
    ctx.close()
