"""The FP32 forms' own arithmetic against 64 bits, on inputs that single out
one rounding or one stencil point each."""
import numpy as np
import pytest

from nimbus_b200 import cuda

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
