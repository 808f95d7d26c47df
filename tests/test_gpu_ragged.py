"""The ragged-pencil kernels (mhd_ragged.cuh) and the general transpose on the
pencil lengths where they can go wrong: every cells-per-thread and image count,
single threads, groups of 8, 16, 32 lanes and of several warps, partial pencil
groups and tiles, arrays that are not 16-byte aligned.  EXACT bit for bit
against the oracle, FAST within the operator tolerance.
"""
import json

import numpy as np
import pytest

from util import GOLDEN, bitwise_equal, rel_l2, sha

pytestmark = pytest.mark.gpu
DT = 0.05
FAST_OP_TOL = 1e-6  # the operator tolerance of test_gpu_ops.py

LENGTHS = [1, 2, 3, 5, 6, 7, 9, 17, 18, 33, 34, 50, 61, 72, 75, 80, 97, 99, 100, 119, 121, 130, 157, 160, 161, 170,
           199, 200, 240, 250, 300, 385, 398, 479, 509, 511]


def state(n, ny, nz, seed, mhd):
    rng = np.random.default_rng(seed)
    u, b = mhd.init_vortex(n, ny, nz, seed=int(rng.integers(1 << 20)))
    u = (u * (1 + 0.05 * rng.standard_normal(u.shape))).astype(np.float32)
    b = (b + 0.05 * rng.standard_normal(b.shape)).astype(np.float32)
    return u, b, (b * np.float32(0.75)).astype(np.float32)


def shifted(torch, a, off):
    """A device copy of `a` that starts `off` floats past a 256-byte boundary."""
    base = torch.zeros(a.size + 64, dtype=torch.float32, device="cuda")
    t = base[off:off + a.size]
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("n", LENGTHS)
def test_ragged_operators_vs_oracle(n, mhd, cuda, oracle32):
    torch = cuda
    for ny, nz, off in ((11, 3, 0), (1, 2, 0), (5, 4, 1)):
        u, b, bin_ = state(n, ny, nz, 100 * n + ny, mhd)
        uo, bo = np.full_like(u, 7), bin_.copy()
        oracle32.fluidx(uo, b.copy(), n, ny, nz, DT, u.copy(), b.copy())
        oracle32.advectbyzx(u.copy(), bo, n, ny, nz, DT, u.copy(), b.copy())
        ut, bt = np.empty_like(u), np.empty_like(b)
        oracle32.transpose12(ut, bt, u.copy(), b.copy(), n, ny, nz)
        for exact in (True, False):
            with mhd.Context(1, 1, 1, exact=exact) as ctx:
                du, db = shifted(torch, u, off), shifted(torch, b, off)
                ou, ob = shifted(torch, np.full_like(u, 7), off), shifted(torch, bin_, off)
                tu, tb = shifted(torch, np.zeros_like(u), off), shifted(torch, np.zeros_like(b), off)
                ctx.op_fluidx(ou, du, db, n, ny, nz, DT)
                ctx.op_advectbyzx(ob, du, db, n, ny, nz, DT)
                ctx.op_transpose12(tu, tb, du, db, n, ny, nz)
                ctx.sync()
                assert ctx.check() == mhd.MHD_OK
                what = (n, ny, nz, off, exact)
                assert bitwise_equal(tu.cpu().numpy(), ut) and bitwise_equal(tb.cpu().numpy(), bt), what
                gu, gb = ou.cpu().numpy(), ob.cpu().numpy()
                if exact:
                    assert bitwise_equal(gu, uo) and bitwise_equal(gb, bo), what
                else:
                    assert rel_l2(gu, uo) < FAST_OP_TOL and rel_l2(gb, bo) < FAST_OP_TOL, what


@pytest.mark.parametrize("n", [96, 128, 256, 512])
def test_unaligned_arrays_of_register_engine_lengths(n, mhd, cuda, oracle32):
    """Lengths with a fixed-length engine, on arrays it cannot take."""
    torch = cuda
    ny, nz = 4, 3
    u, b, bin_ = state(n, ny, nz, n, mhd)
    uo, bo = np.full_like(u, 7), bin_.copy()
    oracle32.fluidx(uo, b.copy(), n, ny, nz, DT, u.copy(), b.copy())
    oracle32.advectbyzx(u.copy(), bo, n, ny, nz, DT, u.copy(), b.copy())
    with mhd.Context(1, 1, 1, exact=True) as ctx:
        du, db = shifted(torch, u, 3), shifted(torch, b, 3)
        ou, ob = shifted(torch, np.full_like(u, 7), 3), shifted(torch, bin_, 3)
        ctx.op_fluidx(ou, du, db, n, ny, nz, DT)
        ctx.op_advectbyzx(ob, du, db, n, ny, nz, DT)
        ctx.sync()
        assert bitwise_equal(ou.cpu().numpy(), uo) and bitwise_equal(ob.cpu().numpy(), bo)


@pytest.mark.parametrize("shape", [(100, 72, 72), (33, 50, 50), (61, 20, 20), (170, 35, 35), (7, 121, 121)])
def test_ragged_steps_vs_oracle(shape, mhd, cuda, oracle32):
    """Plain steps: the side array written by fluidx and by the transposes, the CFL epilogue."""
    u, b = mhd.init_vortex(*shape, seed=9)
    ref = oracle32.strang(u, b, *shape, 3)
    with mhd.Context(*shape, exact=True) as ctx:
        ctx.set_state(u, b)
        ctx.step(3, cfl=0.7)
        gu, gb = ctx.get_state()
        assert ctx.check() == mhd.MHD_OK
        assert bitwise_equal(gu, ref[0]) and bitwise_equal(gb, ref[1])
    with mhd.Context(*shape) as ctx:
        ctx.set_state(u, b)
        ctx.step(3, cfl=0.7)
        gu, gb = ctx.get_state()
        assert rel_l2(gu, ref[0]) < 1e-5 and rel_l2(gb, ref[1]) < 1e-5


# Short pencils and small boxes take one thread per cell, unless the CTAs would hold one short
# pencil each (127 rows, a prime) and be many: the engine's groups of 8 and 16 lanes there.
@pytest.mark.parametrize("n", [n for n in range(3, 41) if n not in (4, 8, 10, 22, 25, 28, 31, 35, 38)])
def test_ragged_short_pencils_in_a_large_box_vs_oracle(n, mhd, cuda, oracle32):
    torch = cuda
    ny, nz = 127, 17
    u, b, bin_ = state(n, ny, nz, 3 * n, mhd)
    uo, bo = np.full_like(u, 7), bin_.copy()
    oracle32.fluidx(uo, b.copy(), n, ny, nz, DT, u.copy(), b.copy())
    oracle32.advectbyzx(u.copy(), bo, n, ny, nz, DT, u.copy(), b.copy())
    for exact in (True, False):
        for off in (0, 1):
            with mhd.Context(1, 1, 1, exact=exact) as ctx:
                du, db = shifted(torch, u, off), shifted(torch, b, off)
                ou, ob = shifted(torch, np.full_like(u, 7), off), shifted(torch, bin_, off)
                ctx.op_fluidx(ou, du, db, n, ny, nz, DT)
                ctx.op_advectbyzx(ob, du, db, n, ny, nz, DT)
                ctx.sync()
                gu, gb = ou.cpu().numpy(), ob.cpu().numpy()
            if exact:
                assert bitwise_equal(gu, uo) and bitwise_equal(gb, bo), off
            else:
                assert rel_l2(gu, uo) < FAST_OP_TOL and rel_l2(gb, bo) < FAST_OP_TOL, off


@pytest.mark.parametrize("edge,boxes", [(15, 64), (18, 40), (20, 10), (21, 24), (30, 8), (33, 6), (40, 4)])
@pytest.mark.parametrize("exact", [False, True])
def test_engine_and_thread_per_cell_give_the_same_steps(edge, boxes, exact, mhd, cuda):
    """A box steps bit for bit alike alone (one thread per cell) and among so many that the
    engine takes them, in both policies."""
    ics = [mhd.init_vortex(edge, edge, edge, seed=s) for s in range(boxes)]
    with mhd.Batch([edge] * boxes, exact=exact) as bt:
        for i, (u, b) in enumerate(ics):
            bt.set_box(i, u, b)
        bt.step(3)
        bt.sync()
        got = [bt.get_box(i) for i in range(boxes)]
    for i in (0, boxes - 1):
        with mhd.Context(edge, edge, edge, exact=exact) as ctx:
            ctx.set_state(*ics[i])
            ctx.step(3)
            u, b = ctx.get_state()
        assert bitwise_equal(got[i][0], u) and bitwise_equal(got[i][1], b)


# FAST on lengths without a fixed engine (the engine and one thread per cell) and on an unaligned
# array of a fixed-engine length: (nx, ny, nz, floats off a 256-byte boundary)
PINNED = [(7, 9, 5, 0), (20, 5, 3, 0), (33, 31, 31, 0), (37, 127, 17, 0), (50, 20, 20, 0), (61, 20, 20, 0),
          (72, 36, 36, 0), (100, 40, 40, 0), (121, 8, 8, 1), (241, 10, 10, 0), (300, 9, 9, 0), (128, 16, 16, 1)]


def pinned_outputs(mhd, torch, n, ny, nz, off) -> str:
    """Digest of one fluidx and one advectbyzx of the seeded vortex in FAST."""
    u, b = mhd.init_vortex(n, ny, nz, seed=n)
    with mhd.Context(1, 1, 1) as ctx:
        du, db = shifted(torch, u, off), shifted(torch, b, off)
        ou, ob = shifted(torch, np.zeros_like(u), off), shifted(torch, (b * np.float32(0.75)), off)
        ctx.op_fluidx(ou, du, db, n, ny, nz, DT)
        ctx.op_advectbyzx(ob, du, db, n, ny, nz, DT)
        ctx.sync()
        return sha(ou.cpu().numpy(), ob.cpu().numpy())


@pytest.mark.parametrize("case", PINNED)
def test_fast_ragged_bits_are_kept(case, mhd, cuda):
    """The bits of the one-thread-per-cell kernels that took these lengths first (a corrected
    run amplifies a last-bit change): digests made with them."""
    want = json.loads((GOLDEN / "fast_ragged.json").read_text())
    assert pinned_outputs(mhd, cuda, *case) == want["%dx%dx%d+%d" % case]


@pytest.mark.parametrize("shape", [(20, 60, 60), (16, 80, 80), (12, 96, 96), (60, 20, 20), (40, 40, 40)])
def test_steps_that_mix_both_kernels_vs_oracle(shape, mhd, cuda, oracle32):
    """Plain steps whose fluidx takes one thread per cell and writes the side array for an
    advectbyzx of the engine, in one sweep or another."""
    u, b = mhd.init_vortex(*shape, seed=3)
    ref = oracle32.strang(u, b, *shape, 2)
    with mhd.Context(*shape, exact=True) as ctx:
        ctx.set_state(u, b)
        ctx.step(2, cfl=0.7)
        gu, gb = ctx.get_state()
        assert ctx.check() == mhd.MHD_OK
    assert bitwise_equal(gu, ref[0]) and bitwise_equal(gb, ref[1])
