"""The FP32 Kessler step's temperature where its power function changes
interval: pressures on both sides of every edge and at the ends of the range,
saturated and cloudy, against the FP64 form (which equals the CPU solver).

Tolerance: the temperature's relative error is a few FP32 roundings, 1e-7; the
saturation vapour pressure multiplies it by L / (R_v T) < 30 and adds the
exponent's own rounding, 20 x 1.2e-7; the adjustment stops at four ulps of the
vapour.  Together below 1e-5 of the vapour content; 2e-5 is allowed."""
import numpy as np
import pytest

from nimbus_b200 import cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cloud", [0.0, 3e-3], ids=["vapour", "cloud"])
@pytest.mark.parametrize("excess", [0.8, 1.3], ids=["dry", "moist"])
def test_saturation_adjustment_across_the_exponents(cloud, excess):
    edges = 1e5 * np.sqrt(0.5) * 2.0 ** np.arange(-5, 2)
    p = np.concatenate([edges * (1 + s) for s in (-1e-3, -1e-7, 0.0, 1e-7, 1e-3)] + [np.geomspace(1e3, 2e5, 189)])
    p = np.sort(p).astype(np.float32).reshape(1, 1, -1).repeat(8, 0).repeat(8, 1)
    exner = (p.astype(np.float64) / 1e5) ** (287.0 / 1004.0)
    T = np.minimum(290.0, 690.0 * exner) - np.linspace(0, 15, 64).reshape(8, 8, 1)
    e = 611.21 * np.exp((18.678 - (T - 273.15) / 234.5) * (T - 273.15) / (257.14 + T - 273.15))
    qv = excess * 0.62198 * e / (p - e)
    st = dict(theta=T / exner, qv=qv, qc=np.full(p.shape, cloud), qr=np.zeros(p.shape), p=p, rho=p / (287.0 * T))
    st = {k: np.ascontiguousarray(v, np.float32) for k, v in st.items()}
    got = []
    ctx = cuda.Context(0)
    for precision in (cuda.PRECISION_FP32, cuda.PRECISION_REFERENCE):
        ctx.set_precision(precision)
        mine = {k: v.copy() for k, v in st.items()}
        ctx.check(ctx.kessler_step(cuda.kessler_args(mine, 300.0, 1e-3)))
        got.append(mine)
    ctx.close()
    for k in ("qv", "qc"):
        off = np.abs(got[0][k].astype(np.float64) - got[1][k]) / np.maximum(st["qv"], st["qc"])
        assert off.max() <= 2e-5, (k, off.max(), p.ravel()[off.argmax() % p.shape[2]])
