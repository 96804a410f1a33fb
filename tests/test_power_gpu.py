"""The equation of state's power in reference precision across the intervals
of its tables: arguments on both sides of every 64th of every octave that the
pressure clamp leaves, against the library power in FP64.  Both are within an
ulp of FP64 of the exact power, so their FP32 results differ only where the
exact value lies that close to the middle of two floats, a chance of 1e-8 a
value; one such value an octave is allowed, by one ulp."""
import numpy as np
import pytest

from nimbus_b200 import cuda
from nimbus_b200.initial import GAMMA, P00, R_D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("octave", range(-5, 1))
def test_pressure_at_every_interval_edge(octave):
    x = 2.0 ** octave * (1 + np.arange(64) / 64)
    x = np.concatenate([x * (1 + s) for s in (-2e-3, -1e-7, 0.0, 1e-7, 5e-8, 2e-3)] * 9)
    rng = np.random.default_rng(octave + 9)
    theta = rng.uniform(230, 450, x.size).astype(np.float32)
    rho = (x * P00 / (R_D * theta)).astype(np.float32)
    shape = (9, 6, 64)
    want = P00 * (rho.astype(np.float64) * R_D * theta / P00) ** GAMMA
    want = np.clip(want.astype(np.float32), np.float32(1000), np.float32(200000))
    p = np.full(shape, 5e4, np.float32)
    ctx = cuda.Context(0)
    ctx.check(ctx.eos_projection(cuda.eos_args(p, rho.reshape(shape), theta.reshape(shape))))
    ctx.close()
    off = np.abs(p.ravel().view(np.int32) - want.view(np.int32))
    assert off.max() <= 1 and np.count_nonzero(off) <= 1, (np.count_nonzero(off), off.max())
