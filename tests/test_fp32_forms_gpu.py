"""The FP32 forms' own arithmetic against 64 bits, on inputs that single out
one rounding or one stencil point each."""
import numpy as np
import pytest

from nimbus_b200 import cuda
from nimbus_b200.initial import Case, perturbed_state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = cuda.Context(0)
    c.set_precision(cuda.PRECISION_FP32)
    yield c
    c.close()


@pytest.mark.parametrize("left", [2.0 ** -4, 2.0 ** -8])
def test_update_of_a_nearly_emptied_cell(ctx, left):
    """A scalar that leaves through one x-face of mass flux M until the
    fraction `left` remains.  dx, dt and M are powers of two and the scalar
    does not vary along x, so the flux and its divergence are exact: the new
    value (rho_b q - dt M q / dx) / rho_e has the rounding of one FMA (half an
    ulp) and of the approximate quotient (two ulps).  Four are allowed; rounding
    rho_b q by itself would add up to half an ulp / `left`."""
    shape, plane, gone = (12, 9, 16), 5, 0.5
    rng = np.random.default_rng(3)
    q = np.broadcast_to(np.exp(rng.uniform(np.log(1e-6), np.log(1e-2), shape[1:])), shape).astype(np.float32)
    rho = (gone * (1 + left * rng.uniform(1, 2, shape))).astype(np.float32)
    zero = np.zeros(shape, np.float32)
    mfx = zero.copy()
    mfx[plane] = gone * 512.0 / 2.0  # dt M / dx = gone
    out = zero.copy()
    ctx.check(ctx.scalar_transport(cuda.transport_args([np.ascontiguousarray(q)], [out], [1], rho, rho, mfx, zero,
                                                       zero, 2.0, (512.0, 512.0, 512.0))))
    want = (rho.astype(np.float64) - gone) * q / rho
    inner = np.s_[plane, 1:-1]
    off = np.abs(out[inner] - want[inner]) / want[inner]
    assert off.max() <= 4 * 2.0 ** -23, off.max()


@pytest.mark.parametrize("sign", [1.0, -1.0], ids=["ahead", "behind"])
@pytest.mark.parametrize("field", ["u", "v", "w"])
def test_slow_tendencies_around_an_infinite_wind(ctx, field, sign):
    """One infinite value: the cells whose stencils hold it have the tendency
    0 (not finite), the ones beside them theirs, as in reference precision; the
    third cell downwind is outside the upwind stencil.  Winds below 13 m/s, so
    a derivative's error is at most 160 / 60 times 13 m/s times four roundings
    over 300 m, below 1e-7, its product with the wind below 2e-6, and three of
    them and the buoyancy's (9.81 m/s2, two roundings) below 1e-5; the
    tendencies are a thousand times that."""
    shape, at = (17, 16, 18), (8, 8, 9)
    case = Case(*shape, 500.0, 450.0, 300.0, 2.0, seed=4)
    st, base = perturbed_state(case, seed=4)
    rng = np.random.default_rng(9)
    for k, mean in (("u", 10.0), ("v", 8.0), ("w", 4.0)):
        st[k] = (sign * mean + rng.uniform(-2, 2, shape)).astype(np.float32)
    st[field][at] = np.inf
    got = {}
    for precision in (cuda.PRECISION_FP32, cuda.PRECISION_REFERENCE):
        ctx.set_precision(precision)
        outs = [np.zeros(shape, np.float32) for _ in range(4)]
        ctx.check(ctx.slow_tendencies(cuda.slow_args(st, base, (case.dx, case.dy, case.dz), outputs=outs)))
        got[precision] = outs
    ctx.set_precision(cuda.PRECISION_FP32)
    for k, mine, want in zip("uvw", got[cuda.PRECISION_FP32], got[cuda.PRECISION_REFERENCE]):
        assert np.count_nonzero(want == 0) < want.size // 2
        off = np.abs(mine - want)
        assert off.max() <= 1e-5, (k, off.max(), np.argwhere(off > 1e-5)[:4].tolist())
