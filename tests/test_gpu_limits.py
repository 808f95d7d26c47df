"""The operators at the limits of the number range, where a form that is equal to the
reference's on ordinary values need not be: sums that overflow, halves and products that
underflow, subnormal densities and pressures, infinities and NaN.  EXACT and FP64 bit
for bit against the oracle (any NaN equals any NaN), FAST within what it can represent.
"""
import zlib

import numpy as np
import pytest

from util import rel_l2

pytestmark = pytest.mark.gpu
DT = 0.05


def same_bits(a, b) -> bool:
    a, b = np.ascontiguousarray(a).copy(), np.ascontiguousarray(b).copy()
    a[np.isnan(a)] = np.nan
    b[np.isnan(b)] = np.nan
    return a.dtype == b.dtype and a.tobytes() == b.tobytes()


def gpu_ops(mhd, torch, u, b, bin_, shape, dt, **mode):
    """(fluidx u, advectbyzx b) of one application each."""
    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda()

    with mhd.Context(1, 1, 1, **mode) as ctx:
        du, db, uo, bo = dev(u), dev(b), dev(np.full_like(u, 7)), dev(bin_)
        ctx.op_fluidx(uo, du, db, *shape, dt)
        ctx.op_advectbyzx(bo, du, db, *shape, dt)
        ctx.sync()
        return uo.cpu().numpy(), bo.cpu().numpy()


def oracle_ops(o, u, b, bin_, shape, dt):
    uo, bo = np.full_like(u, 7), bin_.copy()
    o.fluidx(uo, b.copy(), *shape, dt, u.copy(), b.copy())
    o.advectbyzx(u.copy(), bo, *shape, dt, u.copy(), b.copy())
    return uo, bo


def cells(shape, *key):
    return shape[0] * shape[1] * shape[2], np.random.default_rng(zlib.crc32(repr((shape, key)).encode()))


# one shape for every kernel of advectbyzx (marching, one row per thread, ragged, one thread
# per cell, walking along x)
@pytest.mark.parametrize("shape", [(32, 8, 4), (48, 16, 2), (20, 5, 3), (61, 4, 3), (512, 4, 2)])
def test_exact_face_velocity_near_the_largest_float(shape, mhd, cuda, oracle32):
    """The 1-2-1 smoothing of the face velocity: vm + 2 v + vp passes the largest float
    while its quarter, which the reference takes in double, does not."""
    nc, rng = cells(shape, "v")
    u = np.ones((nc, 5), np.float32)
    u[:, 0] = 0.5
    u[:, 1:4] = 8.4e37 * rng.uniform(0.7, 1, (nc, 3))
    b = (1e-30 * rng.standard_normal((nc, 3))).astype(np.float32).ravel()
    u, bin_ = u.ravel(), (b * np.float32(0.75)).astype(np.float32)
    _, bo = oracle_ops(oracle32, u, b, bin_, shape, 1e-38)
    assert np.isfinite(bo).all() and not np.array_equal(bo, bin_)
    assert same_bits(gpu_ops(mhd, cuda, u, b, bin_, shape, 1e-38, exact=True)[1], bo)


# momenta, energies and fields of 2^lo .. 2^hi around ordinary densities: products of two
# differences underflow (-560), subnormals (-1070), products on the edge of the largest
# double (505), sums beyond it (1000)
@pytest.mark.parametrize("lo,hi", [(-560, -480), (-1070, -1000), (505, 515), (1000, 1023)])
@pytest.mark.parametrize("shape", [(32, 8, 4), (20, 5, 3), (33, 4, 2), (64, 6, 3)])
def test_fp64_operators_at_the_limits(shape, lo, hi, mhd, cuda, oracle64):
    """FP64 keeps the reference's bits where the forms with fewer operations do not hold."""
    nc, rng = cells(shape, lo, hi)
    with np.errstate(over="ignore"):
        u, b, bin_ = (rng.standard_normal((nc, k)) * 2.0 ** rng.uniform(lo, hi, (nc, k)) for k in (5, 3, 3))
    u[:, 0] = 2.0 ** rng.uniform(-3, 3, nc)
    for x in (u[:, 1:], b, bin_):
        x[rng.random(x.shape) < 0.02] = 0
    u, b, bin_ = u.ravel(), b.ravel(), bin_.ravel()
    uo, bo = oracle_ops(oracle64, u, b, bin_, shape, DT)
    gu, gb = gpu_ops(mhd, cuda, u, b, bin_, shape, DT, fp64=True)
    assert same_bits(gu, uo) and same_bits(gb, bo)


@pytest.mark.parametrize("dt", [0.0, 5e-324, 1e-300, 1e300])
def test_fp64_operators_with_extreme_steps(dt, mhd, cuda, oracle64):
    shape = (24, 5, 3)
    nc, rng = cells(shape, dt)
    u, b, bin_ = (rng.standard_normal((nc, k)) for k in (5, 3, 3))
    u[:, 0] = 2.0 ** rng.uniform(-3, 3, nc)
    u, b, bin_ = u.ravel(), b.ravel(), bin_.ravel()
    uo, bo = oracle_ops(oracle64, u, b, bin_, shape, dt)
    gu, gb = gpu_ops(mhd, cuda, u, b, bin_, shape, dt, fp64=True)
    assert same_bits(gu, uo) and same_bits(gb, bo)


# one shape for every kernel of fluidx and advectbyzx
ALL_SHAPES = [(32, 8, 4), (48, 16, 2), (96, 6, 3), (7, 9, 5), (20, 5, 3), (61, 4, 3), (256, 4, 2), (512, 4, 2)]


@pytest.mark.parametrize("shape", ALL_SHAPES)
def test_fast_subnormal_densities(shape, mhd, cuda, oracle32):
    """FAST takes densities below the normal range, 2^-127.5 .. 2^-126.2, with velocities of
    order one: a value of 2^-127 is known to 2^-149, and at most ten such roundings reach a
    cell (dt = 0.05 times some forty of the fluxes, and the sums), 1e-5 of it."""
    nc, rng = cells(shape, "rho")
    rho = 2.0 ** rng.uniform(-127.5, -126.2, nc)
    u = np.empty((nc, 5), np.float32)
    u[:, 0] = rho
    u[:, 1:4] = rho[:, None] * rng.uniform(-1, 1, (nc, 3))
    u[:, 4] = rho * rng.uniform(1, 2, nc)
    b = np.zeros(3 * nc, np.float32)
    bin_ = rng.standard_normal(3 * nc).astype(np.float32)
    u = u.ravel()
    uo, _ = oracle_ops(oracle32, u, b, bin_, shape, DT)
    gu, gb = gpu_ops(mhd, cuda, u, b, bin_, shape, DT)
    assert np.isfinite(gu).all() and rel_l2(gu, uo) < 1e-5
    # the advected field: velocities of order one from these densities
    b = rng.standard_normal(3 * nc).astype(np.float32)
    bin_ = (b * np.float32(0.75)).astype(np.float32)
    _, bo = oracle_ops(oracle32, u, b, bin_, shape, DT)
    _, gb = gpu_ops(mhd, cuda, u, b, bin_, shape, DT)
    assert np.isfinite(gb).all() and rel_l2(gb, bo) < 1e-5


@pytest.mark.parametrize("shape", ALL_SHAPES)
def test_fast_subnormal_pressure(shape, mhd, cuda, oracle32):
    """A gas at rest without field whose pressure over density is subnormal: its sound speed
    is 2^-64, not zero.  Momenta of about 2^-129 within 32 steps of the subnormal grid, the
    energy to 1e-5."""
    nc, rng = cells(shape, "p")
    u = np.zeros((nc, 5), np.float32)
    u[:, 0] = 1
    u[:, 4] = 2.0 ** rng.uniform(-128, -126.5, nc)
    b = np.zeros(3 * nc, np.float32)
    uo, _ = oracle_ops(oracle32, u.ravel(), b, b, shape, DT)
    gu, _ = gpu_ops(mhd, cuda, u.ravel(), b, b, shape, DT)
    assert np.isfinite(gu).all()
    d = gu.reshape(-1, 5).astype(np.float64) - uo.reshape(-1, 5)
    assert np.abs(d[:, 1:4]).max() <= 32 * 2.0 ** -149
    assert np.abs(d[:, 4]).max() <= 1e-5 * u[:, 4].max() and np.array_equal(gu[::5], uo[::5])


@pytest.mark.parametrize("mode", ["f32", "f64"])
@pytest.mark.parametrize("shape", ALL_SHAPES)
def test_infinities_and_nan(shape, mode, mhd, cuda, oracle32, oracle64):
    """One cell in fifty infinite, NaN or a signed zero: the bits of the reference (which
    cells turn NaN or infinite, and all others)."""
    o, dt = (oracle32, np.float32) if mode == "f32" else (oracle64, np.float64)
    nc, rng = cells(shape, mode)
    u, b, bin_ = (rng.standard_normal((nc, k)).astype(dt) for k in (5, 3, 3))
    u[:, 0] = 2.0 ** rng.uniform(-3, 3, nc)
    for x in (u, b, bin_):
        m = rng.random(x.shape) < 0.02 / x.shape[1]
        x[m] = rng.choice(np.array([np.inf, -np.inf, np.nan, 0.0, -0.0], dt), m.sum())
    u, b, bin_ = u.ravel(), b.ravel(), bin_.ravel()
    uo, bo = oracle_ops(o, u, b, bin_, shape, DT)
    gu, gb = gpu_ops(mhd, cuda, u, b, bin_, shape, DT, exact=True, fp64=mode == "f64")
    assert same_bits(gu, uo) and same_bits(gb, bo)
