"""Performance cases of the solver: what is run, on which inputs, and what it should give.

Every case goes through the package's public entry points (the drop-in
operators, ``Context``, ``Batch``, the closure's C ABI and ``Corrector``) on
device arrays.  A pass starts from the case's initial state, so it can be
repeated and its result does not depend on the passes before it.  ``exact``
restates the method in 64 bits with plain torch.
"""
from __future__ import annotations

import json
import math
from pathlib import Path

import numpy as np
import torch

import heterogeneous_mhd_gb300 as mhd
from heterogeneous_mhd_gb300 import closure as cl

CFL = 0.7
GAMMA = 5.0 / 3.0
WEIGHTS = Path(mhd.__file__).resolve().parent / "closure_weights.npz"
FUSED_EDGES = (32, 64, 128, 256)  # pencils the transpose-free sweeps take at every size


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a driver written against the reference's C surface (its main loop, one
        # full Strang step of synchronous operator calls) on a small box: latency
        {"name": "dropin_32", "op": "dropin", "nx": 32, "ny": 32, "nz": 32, "init": "vortex"},
        # the parity configuration: 64^3 vortex, 10 plain Strang steps from an
        # initial state; launch- and latency-bound
        {"name": "plain_64", "op": "step", "variant": "plain", "prec": "f32", "nx": 64, "ny": 64, "nz": 64,
         "steps": 10, "init": "vortex"},
        # a box whose edges are no powers of two (a resolution chosen by physics)
        {"name": "ragged_100x72", "op": "step", "variant": "plain", "prec": "f32", "nx": 100, "ny": 72, "nz": 72,
         "steps": 4, "init": "vortex"},
        # a mid-size production run with the transpose-free step
        {"name": "fused_128", "op": "step", "variant": "fused", "prec": "f32", "nx": 128, "ny": 128, "nz": 128,
         "steps": 10, "init": "turbulence"},
        # the throughput configuration (decaying turbulence), both step variants
        {"name": "plain_256", "op": "step", "variant": "plain", "prec": "f32", "nx": 256, "ny": 256, "nz": 256,
         "steps": 4, "init": "turbulence"},
        {"name": "fused_256", "op": "step", "variant": "fused", "prec": "f32", "nx": 256, "ny": 256, "nz": 256,
         "steps": 4, "init": "turbulence"},
        # the largest box of the configurations
        {"name": "plain_512", "op": "step", "variant": "plain", "prec": "f32", "nx": 512, "ny": 512, "nz": 512,
         "steps": 2, "init": "turbulence"},
        # a parameter study: independent boxes of uneven sizes stepped together
        {"name": "batch_24", "op": "batch", "boxes": 24, "steps": 5, "table": 3},
        # a double-precision run (error studies against the FP32 solver)
        {"name": "fp64_64", "op": "step", "variant": "plain", "prec": "f64", "nx": 64, "ny": 64, "nz": 64,
         "steps": 2, "init": "vortex"},
        # a run that has to reproduce the reference bit for bit
        {"name": "exact_96", "op": "step", "variant": "plain", "prec": "exact", "nx": 96, "ny": 96, "nz": 96,
         "steps": 2, "init": "vortex"},
        # one hidden layer of the closure net in training: forward, data
        # gradient, weight gradient and bias gradient of a batch of boxes
        {"name": "conv_layer_4x64", "op": "layer", "boxes": 4, "n": 64},
        # a coarse run with the trained closure applied after every step
        {"name": "closure_64", "op": "closure", "n": 64, "steps": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["dropin", "plain", "plain", "ragged", "fused", "fused", "batch", "f64", "exact", "layer",
                     "closure"])
    if op == "dropin":
        m = _log_int(rng, 16, 80)
        return {"op": "dropin", "nx": _log_int(rng, 16, 80), "ny": m, "nz": m, "init": "vortex"}
    if op == "plain":  # edges the register-resident kernels were laid out for, not always cubes
        n = rng.choice([32, 48, 64, 96, 128, 192, 256, 384])
        m = rng.choice([e for e in (32, 48, 64, 96, 128, 192, 256, 384) if n * e * e <= 384 ** 3])
        cells = n * m * m
        return {"op": "step", "variant": "plain", "prec": "f32", "nx": n, "ny": m, "nz": m,
                "steps": max(1, min(10, (1 << 27) // cells)), "init": rng.choice(["vortex", "turbulence"])}
    if op == "ragged":
        m = _log_int(rng, 20, 160)
        return {"op": "step", "variant": "plain", "prec": "f32", "nx": _log_int(rng, 20, 240), "ny": m, "nz": m,
                "steps": rng.randint(2, 4), "init": "vortex"}
    if op == "fused":
        nx, ny, nz = rng.choice([32, 64, 96, 128, 160, 256]), rng.choice(FUSED_EDGES), rng.choice(FUSED_EDGES)
        return {"op": "step", "variant": "fused", "prec": "f32", "nx": nx, "ny": ny, "nz": nz,
                "steps": rng.randint(2, 6), "init": rng.choice(["vortex", "turbulence"])}
    if op == "batch":
        return {"op": "batch", "boxes": rng.randint(6, 40), "steps": rng.randint(2, 5), "table": rng.randint(10, 999)}
    if op in ("f64", "exact"):
        m = _log_int(rng, 24, 96 if op == "f64" else 128)
        return {"op": "step", "variant": "plain", "prec": op, "nx": _log_int(rng, 24, 128), "ny": m, "nz": m,
                "steps": rng.randint(1, 3), "init": "vortex"}
    if op == "layer":
        return {"op": "layer", "boxes": rng.randint(1, 6), "n": rng.choice([16, 24, 32, 40, 48, 64])}
    return {"op": "closure", "n": rng.choice([32, 48, 64, 80, 96]), "steps": rng.randint(1, 4)}


# ------------------------------------------------------------- initial states

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _centres(n):
    return (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n


def _energy(rho, p, v, b):
    """Total energy of the cell, with the cell-centred field of the faces b [3][nz][ny][nx]."""
    bc2 = (0.5 * (b[0] + torch.roll(b[0], -1, 2))) ** 2
    bc2 += (0.5 * (b[1] + torch.roll(b[1], -1, 1))) ** 2
    bc2 += (0.5 * (b[2] + torch.roll(b[2], -1, 0))) ** 2
    return p / (GAMMA - 1.0) + 0.5 * rho * (v * v).sum(0) + 0.5 * bc2


def _pack(rho, p, v, b, dtype):
    """(u, b) in the solver's layout: component innermost, x fastest."""
    e = _energy(rho, p, v, b)
    r = torch.full_like(e, rho)
    u = torch.stack([r, rho * v[0], rho * v[1], rho * v[2], e], dim=-1)
    return u.to(dtype).reshape(-1).contiguous(), torch.stack(list(b), dim=-1).to(dtype).reshape(-1).contiguous()


def _vortex(nx, ny, nz, seed, dtype=torch.float32, p0=0.6, vscale=1.0, noise=1e-3):
    """v = (-sin 2 pi y, sin 2 pi x, 0.1 sin 2 pi z) + noise, B = (-sin 2 pi y, sin 4 pi x, 0)/sqrt(4 pi)."""
    f64 = dict(device="cuda", dtype=torch.float64)
    x, y, z = _centres(nx), _centres(ny), _centres(nz)
    tau = 2.0 * math.pi
    v = vscale * noise * torch.randn((3, nz, ny, nx), generator=_gen(seed), **f64)
    v[0] -= vscale * torch.sin(tau * y)[None, :, None]
    v[1] += vscale * torch.sin(tau * x)[None, None, :]
    v[2] += 0.1 * vscale * torch.sin(tau * z)[:, None, None]
    b = torch.zeros((3, nz, ny, nx), **f64)
    b[0] -= (torch.sin(tau * y) / math.sqrt(4.0 * math.pi))[None, :, None]
    b[1] += (torch.sin(2.0 * tau * x) / math.sqrt(4.0 * math.pi))[None, None, :]
    return _pack(1.0, p0, v, b, dtype)


def _random_field(shape, g, power, kmin=2, kmax=8):
    """One Gaussian random field of the modes kmin <= |k| <= kmax with amplitude |k|^-power."""
    nz, ny, nx = shape
    k = torch.cat([torch.arange(0, kmax + 1), torch.arange(1, kmax + 1)]).to("cuda", torch.float32)
    kk = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2)
    amp = torch.where((kk >= kmin) & (kk <= kmax), kk.clamp(min=1.0) ** (-power), torch.zeros_like(kk))
    c = amp * torch.randn(kk.shape, generator=g, device="cuda")

    def basis(n):  # cos(2 pi k x) for k = 0..kmax, then sin for k = 1..kmax
        ph = 2.0 * math.pi * k[:, None] * _centres(n).to(torch.float32)[None, :]
        return torch.cat([torch.cos(ph[:kmax + 1]), torch.sin(ph[kmax + 1:])])

    f = torch.einsum("abc,cx->abx", c, basis(nx))
    f = torch.einsum("abx,by->ayx", f, basis(ny))
    return torch.einsum("ayx,az->zyx", f, basis(nz))


def _turbulence(nx, ny, nz, seed, dtype=torch.float32, mach=0.5, bx0=0.3, dbrms=0.1):
    """Random velocity of rms Mach 0.5 and B = 0.3 x + curl A (discrete, so div B is round-off)."""
    g = _gen(seed)
    shape = (nz, ny, nx)
    v = torch.stack([_random_field(shape, g, 2.0) for _ in range(3)])
    cs = math.sqrt(GAMMA)
    v *= mach * cs / torch.sqrt((v * v).sum(0).mean())
    ax, ay, az = (_random_field(shape, g, 3.0) for _ in range(3))

    def d(a, dim):  # a(i + 1) - a(i)
        return torch.roll(a, -1, dim) - a

    b = torch.stack([d(az, 1) - d(ay, 0), d(ax, 0) - d(az, 2), d(ay, 2) - d(ax, 1)])
    del ax, ay, az
    b *= dbrms / torch.sqrt((b * b).sum(0).mean())
    b[0] += bx0
    return _pack(1.0, 1.0, v, b, dtype)


def _initial(case, seed):
    make = _turbulence if case["init"] == "turbulence" else _vortex
    dtype = torch.float64 if case.get("prec") == "f64" else torch.float32
    return make(case["nx"], case["ny"], case["nz"], seed, dtype)


def _batch_boxes(case, seed):
    """(edge, u, b) of every box: the package's batched workload table, inputs from the seed."""
    out = []
    for i, box in enumerate(mhd.batch_config(case["boxes"], seed=case["table"])):
        p0 = box["beta"] / (8.0 * math.pi)
        vs = box["mach"] * math.sqrt(GAMMA * p0) / math.sqrt(1.005)
        n = box["n"]
        out.append((n, *_vortex(n, n, n, seed * 1009 + i, p0=p0, vscale=vs)))
    return out


# ------------------------------------------------------------- prepare and run

def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op == "dropin":
        s["u0"], s["b0"] = _initial(case, seed)
        for k in ("u", "uu"):
            s[k] = torch.empty_like(s["u0"])
        for k in ("b", "ub"):
            s[k] = torch.empty_like(s["b0"])
    elif op == "step":
        s["u0"], s["b0"] = _initial(case, seed)
        s["ctx"] = mhd.Context(case["nx"], case["ny"], case["nz"], fp64=case["prec"] == "f64",
                               exact=case["prec"] == "exact")
        s["u"], s["b"] = torch.empty_like(s["u0"]), torch.empty_like(s["b0"])
    elif op == "batch":
        s["boxes"] = _batch_boxes(case, seed)
        s["batch"] = mhd.Batch([n for n, _, _ in s["boxes"]])
        # results: four groups of boxes (every fourth box), each group's arrays one after the other
        s["out"] = [None] * len(s["boxes"])
        s["groups"] = []
        for k in range(min(4, len(s["boxes"]))):
            ids = range(k, len(s["boxes"]), 4)
            cells = [s["boxes"][i][0] ** 3 for i in ids]
            u, b = (torch.empty(c * sum(cells), device="cuda") for c in (5, 3))
            for i, uv, bv in zip(ids, u.split([5 * c for c in cells]), b.split([3 * c for c in cells])):
                s["out"][i] = (uv, bv)
            s["groups"].append({"u": u, "b": b})
    elif op == "layer":
        nb, n = case["boxes"], case["n"]
        nv = nb * n ** 3
        g = _gen(seed)
        bf = dict(device="cuda", dtype=torch.bfloat16)
        s["w"] = torch.randn(32 * 27 * 32, generator=g, device="cuda") * math.sqrt(2.0 / (32 * 27))
        s["bias"] = 0.1 * torch.randn(32, generator=g, device="cuda")
        for k, scale in (("a", 1.0), ("dz", 1e-3), ("zprev", 1.0)):
            s[k] = (scale * torch.randn(nv * 32, generator=g, device="cuda")).to(torch.bfloat16)
        s["wf"], s["wd"] = torch.empty(32 * 27 * 32, **bf), torch.empty(32 * 27 * 32, **bf)
        s["y"], s["z"], s["dx"] = (torch.empty(nv * 32, **bf) for _ in range(3))
        s["dw"] = torch.empty(32 * 27 * 32, device="cuda")
        s["db"] = torch.empty(32, device="cuda")
        ws = int(cl.cl().mhd_cl_wgrad_scratch(cl.WG_HID, nb, n))
        s["wsc"] = torch.empty(ws // 4 + 1, device="cuda")
        s["csc"] = torch.empty(256 * 32, device="cuda")
        mhd._check(cl.cl().mhd_cl_pack(s["w"].data_ptr(), 32, 32, 27, 32, 32, s["wf"].data_ptr(),
                                       s["wd"].data_ptr(), cl.stream_ptr()), "mhd_cl_pack")
    elif op == "closure":
        n = case["n"]
        s["u0"], s["b0"] = _vortex(n, n, n, seed)
        s["ctx"] = mhd.Context(n, n, n)
        s["corr"] = cl.Corrector(cl.ClosureNet.load(WEIGHTS), n)
        s["stream"] = torch.cuda.ExternalStream(s["ctx"].stream())
        s["u"], s["b"] = torch.empty_like(s["u0"]), torch.empty_like(s["b0"])
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "dropin":
        return _run_dropin(s)
    if op == "step":
        ctx = s["ctx"]
        ctx.set_state(s["u0"], s["b0"])
        ctx.step(case["steps"], cfl=CFL, fused=case["variant"] == "fused")
        ctx.get_state_into(s["u"], s["b"])
        return {"u": s["u"], "b": s["b"]}
    if op == "batch":
        bt = s["batch"]
        for i, (_, u, b) in enumerate(s["boxes"]):
            bt.set_box(i, u, b)
        bt.step(case["steps"], cfl=CFL)
        for i, (u, b) in enumerate(s["out"]):
            bt.get_box_into(i, u, b)
        return s["groups"]
    if op == "layer":
        L, st, nb, n = cl.cl(), cl.stream_ptr(), case["boxes"], case["n"]
        p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
        mhd._check(L.mhd_cl_conv(cl.FWD_HID, p["a"], p["wf"], p["bias"], p["y"], p["z"], None, nb, n, st), "forward")
        mhd._check(L.mhd_cl_wgrad(cl.WG_HID, p["a"], p["dz"], p["wsc"], p["dw"], nb, n, st), "weight gradient")
        mhd._check(L.mhd_cl_colsum(p["dz"], 32, nb * n ** 3, 32, p["csc"], p["db"], st), "bias gradient")
        mhd._check(L.mhd_cl_conv(cl.DGRAD_HID, p["dz"], p["wd"], None, p["dx"], None, p["zprev"], nb, n, st),
                   "data gradient")
        return {k: s[k] for k in ("y", "z", "dx", "dw", "db")}
    ctx, corr = s["ctx"], s["corr"]
    ctx.set_state(s["u0"], s["b0"])
    up, bp = ctx.state_ptrs()
    with torch.cuda.stream(s["stream"]):  # the solver's own stream: everything in order
        for _ in range(case["steps"]):
            corr.predict(up, bp)
            ctx.step(1, cfl=CFL)
            corr.apply(up, bp)
    ctx.get_state_into(s["u"], s["b"])
    return {"u": s["u"], "b": s["b"]}


def _run_dropin(s):
    """The reference's main loop (C/mhd.c), one step: every operator reads the copies uu, ub."""
    nx, ny, nz = (s["case"][k] for k in ("nx", "ny", "nz"))
    u, b, uu, ub = s["u"], s["b"], s["uu"], s["ub"]
    mhd.copy_matrix(s["u0"], s["b0"], nx, ny, nz, u, b)
    mhd.copy_matrix(u, b, nx, ny, nz, uu, ub)
    dt = CFL * mhd.calcfl(u, b, nx, ny, nz)
    x, y, z = (nx, ny, nz), (ny, nx, nz), (nz, nx, ny)
    for name, d in (("f", x), ("a", x), ("t12", x), ("f", y), ("a", y), ("t13", y), ("f", z), ("a", z), ("a", z),
                    ("f", z), ("t13", z), ("a", y), ("f", y), ("t12", y), ("a", x), ("f", x)):
        if name == "f":
            mhd.fluidx(u, b, *d, dt, uu, ub)
        elif name == "a":
            mhd.advectbyzx(u, b, *d, dt, uu, ub)
        elif name == "t12":
            mhd.transpose12(u, b, uu, ub, *d)
            d = (d[1], d[0], d[2])
        else:
            mhd.transpose13(u, b, uu, ub, *d)
            d = (d[2], d[1], d[0])
        mhd.copy_matrix(u, b, *d, uu, ub)
    return {"u": u, "b": b}


# ------------------------------------------------------------------- the work

def work(case):
    op = case["op"]
    if op == "layer":
        nv = case["boxes"] * case["n"] ** 3
        # a, dz, zprev in; y, z, dx out (BF16), weights and their gradient
        return {"bytes": 6 * nv * 64 + 3 * 27648 * 4, "flops": 3 * 2 * nv * 27 * 32 * 32}
    per_cell = 6 * 330 + 6 * 95 + 25  # six fluidx, six advectbyzx, one CFL speed
    if op == "dropin":
        # every call reads its inputs and writes its outputs: 6 fluidx (52 bytes
        # a cell), 6 advectbyzx (44), 4 transposes and 18 copies (64), calcfl (32)
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": cells * (6 * 52 + 6 * 44 + 22 * 64 + 32), "flops": cells * per_cell}
    if op == "batch":
        cells = sum(b["n"] ** 3 for b in mhd.batch_config(case["boxes"], seed=case["table"])) * case["steps"]
        return {"bytes": cells * 64, "flops": cells * per_cell}
    if op == "closure":
        cells = case["n"] ** 3 * case["steps"]
        net = 2 * (27 * 8 * 32 + 3 * 27 * 32 * 32 + 32 * 8)
        return {"bytes": cells * 128, "flops": cells * (per_cell + net)}
    # a step's dt needs the whole state, so every step reads and writes it once
    cells = case["nx"] * case["ny"] * case["nz"] * case["steps"]
    return {"bytes": cells * (128 if case["prec"] == "f64" else 64), "flops": cells * per_cell}


# ------------------------------------------------- the same in 64 bits, plain torch

def _vanleer(a, b):
    ab = a * b
    s = a + b
    return torch.where(ab > 0, 2.0 * ab / torch.where(ab > 0, s, torch.ones_like(s)), torch.zeros_like(ab))


def _flux(q, f):
    """Fluxes along the sweep and the fast speed of every cell; q = (rho, m_d, m_j, m_k, E)."""
    vx = q[1] / q[0]
    mm = q[1] ** 2 + q[2] ** 2 + q[3] ** 2
    bb = f[0] ** 2 + f[1] ** 2 + f[2] ** 2
    ps = (q[4] - 0.5 * mm / q[0]) * (GAMMA - 1.0) + (2.0 - GAMMA) * 0.5 * bb
    v = [q[1], q[1] * vx + ps - f[0] * f[0], q[2] * vx - f[1] * f[0], q[3] * vx - f[2] * f[0],
         (q[4] + ps) * vx - f[0] * (f[0] * q[1] + f[1] * q[2] + f[2] * q[3]) / q[0]]
    p = ps - 0.5 * bb
    return v, vx.abs() + torch.sqrt(((bb + GAMMA * p) / q[0]).abs())


# per axis: the array dimension of the sweep and of its two neighbours, and the
# components seen along (sweep, j, k); arrays are [component][z][y][x]
_AXES = {0: ((2, 1, 0), (1, 2, 3), (0, 1, 2)), 1: ((1, 2, 0), (2, 1, 3), (1, 0, 2)),
         2: ((0, 2, 1), (3, 1, 2), (2, 0, 1))}


def _fluidx64(u, b, axis, dt):
    (dd, dj, dk), (md, mj, mk), (bd, bj, bk) = _AXES[axis]

    def up(a):  # a(i + 1)
        return torch.roll(a, -1, dd)

    def dn(a):
        return torch.roll(a, 1, dd)

    f = [0.5 * (b[bd] + up(b[bd])), 0.5 * (b[bj] + torch.roll(b[bj], -1, dj)),
         0.5 * (b[bk] + torch.roll(b[bk], -1, dk))]
    order = (0, md, mj, mk, 4)
    q = [u[c] for c in order]
    v, ci = _flux(q, f)
    c = ci.amax(dim=dd, keepdim=True)
    q1 = []
    for s in range(5):
        fl = 0.5 * ((c * q[s] + v[s]) - up(c * q[s] - v[s]))
        q1.append(q[s] - 0.5 * dt * (fl - dn(fl)))
    v, ci = _flux(q1, f)
    c = ci.amax(dim=dd, keepdim=True)
    out = [None] * 5
    for s in range(5):
        fr, gl = c * q1[s] + v[s], c * q1[s] - v[s]
        gn = up(gl)
        dfm, dlm = 0.5 * (fr - dn(fr)), 0.5 * (gl - gn)
        fl = 0.5 * ((fr - gn) + (_vanleer(up(dfm), dfm) - _vanleer(up(dlm), dlm)))
        out[order[s]] = q[s] - dt * (fl - dn(fl))
    return out


def _tvdb64(vf, b, dt, dd):
    """One advected component: its new value and the flux through the face i + 1/2."""

    def up(a, n=1):
        return torch.roll(a, -n, dd)

    def dn(a):
        return torch.roll(a, 1, dd)

    vg = 0.25 * (dn(vf) + up(vf) + 2.0 * vf)
    vh = 0.5 * (vg + up(vg))
    w = b * vg
    f1 = torch.where(vh > 0, w, up(w))
    vb = vg * (b - 0.5 * dt * (f1 - dn(f1)))
    pos = vh > 0
    wc = torch.where(pos, vb, up(vb))
    wp = 0.5 * torch.where(pos, up(vb) - vb, up(vb) - up(vb, 2))
    wm = 0.5 * torch.where(pos, vb - dn(vb), vb - up(vb))
    fx = (wc + _vanleer(wm, wp)) * dt
    return b - (fx - dn(fx)), fx


def _advect64(u, b, axis, dt):
    (dd, dj, dk), (md, _, _), (bd, bj, bk) = _AXES[axis]
    out = list(b)
    new = b[bd]
    for dim, comp in ((dj, bj), (dk, bk)):
        vf = (torch.roll(u[md], 1, dim) + u[md]) / (torch.roll(u[0], 1, dim) + u[0])
        out[comp], fx = _tvdb64(vf, b[comp], dt, dd)
        fm = torch.roll(fx, 1, dd)
        new = new - fm + torch.roll(fm, -1, dim)
    out[bd] = new
    return out


def _dt64(u, b):
    v = torch.maximum(torch.maximum(u[1].abs(), u[2].abs()), u[3].abs()) / u[0]
    mm, bb = u[1] ** 2 + u[2] ** 2 + u[3] ** 2, b[0] ** 2 + b[1] ** 2 + b[2] ** 2
    p = (u[4] - 0.5 * mm / u[0]) * (GAMMA - 1.0) + (2.0 - GAMMA) * 0.5 * bb - 0.5 * bb
    return CFL / (v + torch.sqrt((2.0 * bb + GAMMA * p).abs() / u[0])).max()


def _strang64(u, b, steps=1):
    for _ in range(steps):
        dt = _dt64(u, b)
        for what, axis in (("f", 0), ("a", 0), ("f", 1), ("a", 1), ("f", 2), ("a", 2), ("a", 2), ("f", 2), ("a", 1),
                           ("f", 1), ("a", 0), ("f", 0)):
            if what == "f":
                u = _fluidx64(u, b, axis, dt)
            else:
                b = _advect64(u, b, axis, dt)
    return u, b


def _planes(a, nx, ny, nz, comps):
    return [t.contiguous() for t in a.double().reshape(nz, ny, nx, comps).unbind(-1)]


def _flat(parts):
    return torch.stack(list(parts), dim=-1).reshape(-1)


def _run64(u, b, nx, ny, nz, steps):
    u, b = _strang64(_planes(u, nx, ny, nz, 5), _planes(b, nx, ny, nz, 3), steps)
    return {"u": _flat(u), "b": _flat(b)}


def _shifted(x, dk, dj, di):
    return torch.roll(x, (-dk, -dj, -di), (1, 2, 3))


_TAPS = [(k, j, i) for k in (-1, 0, 1) for j in (-1, 0, 1) for i in (-1, 0, 1)]


def _conv64(x, w):
    """x [boxes][n][n][n][cin], w [cout][27][cin]: the periodic 3^3 convolution."""
    return sum(_shifted(x, *t) @ w[:, q, :].T for q, t in enumerate(_TAPS))


def _gelu64(z):
    return 0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0)))


def _gelu_grad64(z):
    return 0.5 * (1.0 + torch.erf(z / math.sqrt(2.0))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi)


def _exact_layer(case, seed):
    s = prepare(case, seed)
    nb, n = case["boxes"], case["n"]
    shape = (nb, n, n, n, 32)
    a, dz, zp = (s[k].double().reshape(shape) for k in ("a", "dz", "zprev"))
    w = s["w"].to(torch.bfloat16).double().reshape(32, 27, 32)
    z = _conv64(a, w) + s["bias"].double()
    dx = sum(_shifted(dz, *(-c for c in t)) @ w[:, q, :] for q, t in enumerate(_TAPS)) * _gelu_grad64(zp)
    rows = dz.reshape(-1, 32).T
    dw = torch.stack([rows @ _shifted(a, *t).reshape(-1, 32) for t in _TAPS], dim=1)
    return {"y": _gelu64(z).reshape(-1), "z": z.reshape(-1), "dx": dx.reshape(-1), "dw": dw.reshape(-1),
            "db": dz.reshape(-1, 32).sum(0)}


def _exact_closure(case, seed):
    """Net on the state before the step, plain step, then the first of the full, half and
    quarter corrections that keeps rho and p positive and the energy within 1e-3."""
    n = case["n"]
    with np.load(WEIGHTS) as f:
        flat = torch.from_numpy(f["params"].astype(np.float64)).cuda()
        meta = json.loads(bytes(f["meta"]).decode())
    st = meta["stats"]
    gain = meta["gain_by_edge"].get(str(n), meta["gain"])
    mean, inv = (torch.tensor(st[k], dtype=torch.float64, device="cuda") for k in ("mean", "inv_std"))
    layers, o = [], 0
    for cout, cin, taps in ((32, 8, 27), (32, 32, 27), (32, 32, 27), (32, 32, 27), (8, 32, 1)):
        w = flat[o:o + cout * taps * cin].reshape(cout, taps, cin)
        o += cout * taps * cin
        layers.append((w, flat[o:o + cout]))
        o += cout

    def centred(b):
        return [0.5 * (b[c] + torch.roll(b[c], -1, 2 - c)) for c in range(3)]

    u, b = _vortex(n, n, n, seed)
    u, b = _planes(u, n, n, n, 5), _planes(b, n, n, n, 3)
    for _ in range(case["steps"]):
        x = ((torch.stack(list(u) + centred(b), dim=-1) - mean) * inv)[None]
        for w, bias in layers[:-1]:
            x = _gelu64(_conv64(x, w) + bias)
        out = (x[0] @ layers[-1][0][:, 0, :].T + layers[-1][1]).unbind(-1)
        u, b = _strang64(u, b)
        ex, ey, ez = out[5:]

        def d(a, axis):
            return torch.roll(a, -1, 2 - axis) - a

        curl = (-d(ez, 1) + d(ey, 2), -d(ex, 2) + d(ez, 0), -d(ey, 0) + d(ex, 1))
        for alpha in (1.0, 0.5, 0.25):
            uc = [u[c] + alpha * gain * st["oscale"][c] * (out[c] - out[c].mean()) for c in range(5)]
            bc = [b[c] + alpha * gain * st["bscale"] * curl[c] for c in range(3)]
            bb = sum(f * f for f in centred(bc))
            p = (GAMMA - 1.0) * (uc[4] - 0.5 * (uc[1] ** 2 + uc[2] ** 2 + uc[3] ** 2) / uc[0] - 0.5 * bb)
            energy_ok = (uc[4].sum() - u[4].sum()).abs() <= 1e-3 * u[4].sum().abs()
            if bool((uc[0] > 0).all() & (p > 0).all() & energy_ok):
                u, b = uc, bc
                break
    return {"u": _flat(u), "b": _flat(b)}


def exact(case, seed):
    op = case["op"]
    if op == "layer":
        return _exact_layer(case, seed)
    if op == "closure":
        return _exact_closure(case, seed)
    if op == "batch":
        got = [_run64(u, b, n, n, n, case["steps"]) for n, u, b in _batch_boxes(case, seed)]
        return [{k: torch.cat([r[k] for r in got[q::4]]) for k in ("u", "b")} for q in range(min(4, len(got)))]
    u, b = _initial(case, seed)
    return _run64(u, b, case["nx"], case["ny"], case["nz"], case.get("steps", 1))
