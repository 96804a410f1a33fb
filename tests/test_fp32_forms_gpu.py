"""The FP32 forms' own arithmetic against 64 bits, on inputs that single out
one rounding or one stencil point each."""
import numpy as np
import pytest
import torch

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


@pytest.mark.parametrize("way", [1.0, -1.0], ids=["west-outflow", "west-inflow"])
def test_update_beside_a_density_that_is_not_finite(ctx, way):
    """A boundary cell whose old density is -infinity and that gives to another
    boundary cell has a limiter factor that is not finite.  The cell beside it loses its value if it takes from there,
    and keeps it if it gives: to a few roundings of reference precision
    (1e-5 is allowed)."""
    shape, edge = (9, 8, 10), (0, 4, 5)
    rng = np.random.default_rng(6)
    q = rng.uniform(1e-3, 1e-2, shape).astype(np.float32)
    rho = rng.uniform(0.8, 1.0, shape).astype(np.float32)
    begin = rho.copy()
    begin[edge] = -np.inf
    zero = np.zeros(shape, np.float32)
    mfx, mfy = np.full(shape, -5.0 * way, np.float32), zero.copy()
    mfy[edge] = 2.0
    got, codes = [], []
    for precision in (cuda.PRECISION_FP32, cuda.PRECISION_REFERENCE):
        ctx.set_precision(precision)
        out = np.zeros(shape, np.float32)
        codes.append(ctx.scalar_transport(cuda.transport_args([q], [out], [1], rho, begin, mfx, mfy, zero, 2.0,
                                                              (500.0, 500.0, 300.0))))
        got.append(out)
    ctx.set_precision(cuda.PRECISION_FP32)
    assert codes[0] == codes[1]
    if way > 0:
        assert codes[0] == 0
        np.testing.assert_allclose(got[0][1:-1, 1:-1], got[1][1:-1, 1:-1], rtol=1e-5)
    else:
        assert codes[0] != 0


def test_update_takes_in_an_infinite_scalar(ctx):
    """What flows in from an infinite value on the boundary is infinite, not
    undefined, as in reference precision (the step's rain evaporates by it)."""
    shape, edge = (9, 8, 10), (0, 4, 5)
    rng = np.random.default_rng(6)
    q = rng.uniform(1e-3, 1e-2, shape).astype(np.float32)
    q[edge] = np.inf
    rho = rng.uniform(0.8, 1.0, shape).astype(np.float32)
    q, rho, mfx, zero = (torch.from_numpy(x).cuda() for x in (q, rho, np.full(shape, 5.0, np.float32),
                                                             np.zeros(shape, np.float32)))
    for precision in (cuda.PRECISION_REFERENCE, cuda.PRECISION_FP32):
        ctx.set_precision(precision)
        out = torch.zeros(shape, device="cuda")
        torch.cuda.synchronize()
        ctx.check(ctx.scalar_transport(cuda.transport_args([q], [out], [1], rho, rho, mfx, zero, zero, 2.0,
                                                           (500.0, 500.0, 300.0), memory=cuda.MEMORY_DEVICE)))
        with pytest.raises(RuntimeError, match="NONFINITE"):
            ctx.synchronize()
        assert out[1, 4, 5] == np.inf, precision


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


@pytest.mark.parametrize("sign", [1.0, -1.0], ids=["ahead", "behind"])
@pytest.mark.parametrize("axis,field", [(0, "u"), (1, "v"), (2, "w")])
def test_slow_tendencies_behind_a_huge_wind(ctx, axis, field, sign):
    """One wind of 1e38 m/s, two and three cells downwind: the first enters the
    derivative three times, the second not at all, and no sum on the way
    overflows that the tendency does not.  The tendencies (up to 1e36) agree
    with reference precision to a few roundings (1e-6 of the value; 1e-5 is
    allowed, and 1e-5 as beside an infinite wind)."""
    shape, at = (17, 16, 18), np.array((8, 8, 9))
    case = Case(*shape, 500.0, 450.0, 300.0, 2.0, seed=4)
    st, base = perturbed_state(case, seed=4)
    rng = np.random.default_rng(9)
    for k, mean in (("u", 10.0), ("v", 8.0), ("w", 4.0)):
        st[k] = (sign * mean + rng.uniform(-2, 2, shape)).astype(np.float32)
    st[field][tuple(at)] = 1e38
    got = []
    for precision in (cuda.PRECISION_FP32, cuda.PRECISION_REFERENCE):
        ctx.set_precision(precision)
        outs = [np.zeros(shape, np.float32) for _ in range(4)]
        ctx.check(ctx.slow_tendencies(cuda.slow_args(st, base, (case.dx, case.dy, case.dz), outputs=outs)))
        got.append(outs[axis])
    ctx.set_precision(cuda.PRECISION_FP32)
    for away in (2, 3):
        cell = at.copy()
        cell[axis] -= int(sign) * away
        mine, want = (float(g[tuple(cell)]) for g in got)
        assert (abs(want) > 1e34) == (away == 2)
        assert abs(mine - want) <= 1e-5 * abs(want) + 1e-5, (away, mine, want)


def _weno_offsets(v, real, fma):
    """The normalised WENO5-JS offset from the donor v[2], every weight by its
    own reciprocal, in `real` arithmetic with a fused multiply-add."""
    a, b, c, d, e = (x.astype(real) for x in v)
    scale = np.maximum.reduce([abs(x) for x in (a, b, c, d, e)])
    inv = real(1) / scale
    a, b, d, e = ((x - c) * inv for x in (a, b, d, e))
    third, sixth = real(1 / 3), real(1 / 6)
    p = (fma(a, third, b * real(-7 / 6)), fma(d, third, b * -sixth), fma(d, real(5 / 6), e * -sixth))
    smooth = [fma(x * real(13 / 12), x, y * real(0.25) * y)
              for x, y in ((fma(b, real(-2), a), fma(b, real(-4), a)), (b + d, b - d),
                           (fma(d, real(-2), e), fma(d, real(-4), e)))]
    relative = (scale * inv)
    eps = relative * real(1e-6) * relative
    r = [real(1) / (eps + s) for s in smooth]
    w = [x * real(g) * x for x, g in zip(r, (0.1, 0.6, 0.3))]
    return scale, fma(w[2], p[2], fma(w[1], p[1], w[0] * p[0])) / (w[0] + w[1] + w[2]) * scale


def test_weno_offsets_of_resolved_waves(ctx):
    """WENO5 offsets of waves of 12 to 60 cells about an empty donor, whose
    flux is M times the offset and whose only face with a mass flux is read
    off the update (dx, dt, M and the density are powers of two: no rounding).
    The mean square error against 64 bits, relative to the stencil's largest
    value, is at most 5 % above that of the same formula with each weight by
    its own reciprocal and every operation correctly rounded: the normalising
    reciprocal is approximate (an ulp, not half), which is a quarter of the
    squared error and grows by less than a fifth; the rest may not grow."""
    rows, plane = 64, 5
    shape = (12, rows + 2, 256)
    rng = np.random.default_rng(12)
    x = np.arange(12).reshape(12, 1, 1) - plane
    length, phase = np.exp(rng.uniform(np.log(12), np.log(60), shape[1:])), rng.uniform(0, 7, shape[1:])
    size = np.exp(rng.uniform(-9, 0, shape[1:]))
    q = (size * (np.sin(2 * np.pi * x / length + phase) - np.sin(phase))).astype(np.float32)
    half, zero = np.full(shape, 0.5, np.float32), np.zeros(shape, np.float32)
    mfx, out = zero.copy(), zero.copy()
    mfx[plane] = 0.5
    ctx.check(ctx.scalar_transport(cuda.transport_args([np.ascontiguousarray(q)], [out], [0], half, half, mfx, zero,
                                                       zero, 1.0, (1.0, 1.0, 1.0))))
    stencil = [np.ascontiguousarray(q[plane + o, 1:-1]) for o in (-2, -1, 0, 1, 2)]

    def fma32(a, b, c):
        return (a.astype(np.float64) * np.float64(b) + c.astype(np.float64)).astype(np.float32)

    scale, exact = _weno_offsets(stencil, np.float64, lambda a, b, c: a * b + c)
    _, rounded = _weno_offsets(stencil, np.float32, fma32)
    mine = -out[plane, 1:-1]  # 0 - dt (M offset) / dx / rho
    error = [np.sqrt(np.mean(((v - exact) / scale) ** 2)) for v in (mine.astype(np.float64), rounded)]
    assert error[0] <= 1.05 * error[1], error
