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
