"""Performance cases of the MHD stage: what a solver built on this package has it do, through GodunovImplemGB300.

A case names the entry point ("call"), the problem, the mesh and the options:

  step     do_time_step: one stage of a solver that keeps its own loop
  inv_dt   compute_inv_dt: the CFL reduction of such a loop
  advance  the solver loop on the device, `steps` iterations (restarted from the same state on each pass, as a
           parameter study does)
  host     step_host: one stage on page-locked host arrays
  regrid   one AMR cycle (flags, adapt, remap, tables) from the same mesh on each pass

Meshes are uniform leaves of a brick forest (`level` refinements, `bricks` root trees along x), a statically
refined two- or three-level mesh (the blast's front, the shear layers), or a batch of independent problems.
"""
import math
import random

import numpy as np
import torch

from godunov_mhd_ct_gb300 import workloads
from godunov_mhd_ct_gb300.mesh import BlockMesh
from godunov_mhd_ct_gb300.settings import MHDSettings
from godunov_mhd_ct_gb300.solver import GodunovImplemGB300

DEFAULTS = {"dim": 3, "level": 1, "max_level": 0, "bricks": 1, "block": 16, "precision": "mixed", "steps": 1,
            "slope_type": 2.0, "mu": 0.0, "gravity": 0.0, "integrator": "HANCOCK", "problems": 1, "walls": False}


def listed():
    return [
        # the 2D Orszag-Tang vortex on 128^2 cells, FP64: a solver's own loop on a small problem
        {"name": "ot2d_fp64_step", "call": "step", "problem": "ot", "dim": 2, "level": 3, "precision": "fp64"},
        # the same problem in the solver loop, mixed precision: launches and latency
        {"name": "ot2d_mixed_advance", "call": "advance", "problem": "ot", "dim": 2, "level": 3, "steps": 20},
        # a single stage on 32^3 cells: the smallest 3D call
        {"name": "ot3d_small_mixed_step", "call": "step", "problem": "ot", "dim": 3, "level": 1},
        # the FP64 drop-in in 3D
        {"name": "ot3d_fp64_step", "call": "step", "problem": "ot", "dim": 3, "level": 2, "block": 32,
         "precision": "fp64"},
        # 3D Orszag-Tang 256^3 in blocks of 32^3, mixed: the headline workload
        {"name": "ot3d_mixed_step", "call": "step", "problem": "ot", "dim": 3, "level": 3, "block": 32},
        # the CFL reduction that a solver with its own loop does before each of those steps
        {"name": "ot3d_inv_dt", "call": "inv_dt", "problem": "ot", "dim": 3, "level": 3, "block": 32},
        # viscosity and gravity, mixed, 128^3
        {"name": "ot3d_sources_mixed_step", "call": "step", "problem": "ot", "dim": 3, "level": 2, "block": 32,
         "mu": 1e-3, "gravity": 0.1},
        # a state kept in host memory, 128^3
        {"name": "ot3d_host_step", "call": "host", "problem": "ot", "dim": 3, "level": 2, "block": 32},
        # 2D magnetised blast on a coarse/fine mesh: the ten steps between two AMR cycles
        {"name": "blast_amr_mixed_advance", "call": "advance", "problem": "blast", "dim": 2, "level": 5, "max_level": 8,
         "steps": 10},
        # the AMR cycle of that run
        {"name": "blast_amr_regrid", "call": "regrid", "problem": "blast", "dim": 2, "level": 5, "max_level": 8},
        # 3D magnetised shear layers on a coarse/fine mesh with reflecting walls in y
        {"name": "kh3d_amr_mixed_advance", "call": "advance", "problem": "kh", "dim": 3, "level": 3, "max_level": 4,
         "steps": 2, "walls": True},
        # independent field loops of uneven sizes in one batch, each with its own time step
        {"name": "loops_mixed_advance", "call": "advance", "problem": "loops", "dim": 2, "problems": 96, "steps": 10},
    ]


def draw(rng: random.Random):
    c = {"dim": rng.choice([2, 3, 3]), "precision": rng.choice(["mixed", "mixed", "fp64"]),
         "slope_type": rng.choice([1.0, 2.0])}
    kind = rng.choice(["step", "step", "advance", "inv_dt", "host", "amr", "loops"])
    wide = c["precision"] == "mixed"  # an FP64 stage costs some fifty times a mixed one: smaller sizes
    if kind == "amr":
        if c["dim"] == 2:
            lo = rng.choice([3, 4, 5] if wide else [3, 4])
            c.update(call=rng.choice(["advance", "step", "regrid"]), problem="blast", level=lo,
                     max_level=lo + rng.choice([1, 2, 3]), block=rng.choice([8, 16]), steps=rng.randint(2, 10 if wide else 3))
        else:
            c.update(call=rng.choice(["advance", "step"]), problem="kh", level=2, max_level=3,
                     block=rng.choice([8, 12, 16, 20] if wide else [8, 12]), steps=rng.randint(2, 5) if wide else 2,
                     walls=rng.random() < 0.5)
        return c
    if kind == "loops":
        most = math.log(96 if wide else 12)
        c.update(call="advance", problem="loops", dim=2, problems=int(round(math.exp(rng.uniform(math.log(4), most)))),
                 steps=rng.randint(2, 10 if wide else 4))
        return c
    # uniform meshes: cells spread over their logarithm, up to 128^3 in FP64 and 256^3 in mixed precision
    c.update(steps=rng.randint(1, 4) if kind == "advance" else 1,
             integrator=rng.choice(["HANCOCK", "HANCOCK", "RK2_SSP"]) if kind == "advance" else "HANCOCK")
    block = rng.choice([8, 12, 16, 16, 20, 24, 32, 32, 36])
    top = math.log((2.0 ** 24 if (wide and kind != "host") or kind == "inv_dt" else 2.0 ** 21)
                   / (c["steps"] * (2 if c["integrator"] == "RK2_SSP" else 1)))
    want = math.exp(rng.uniform(math.log(2.0 ** 13), top))
    bricks, level, best = 1, 0, None
    for b in (1, 2, 3):
        for lv in range(0, 9 if c["dim"] == 2 else 5):
            cells = b * (block << lv) ** c["dim"]
            if cells > 1.2 * math.exp(top):
                continue
            miss = abs(math.log(cells / want))
            if best is None or miss < best:
                best, bricks, level = miss, b, lv
    c.update(call=kind, problem=rng.choice(["ot", "blast"]), block=block, bricks=bricks, level=level)
    if kind != "inv_dt":
        if rng.random() < 0.2:
            c["mu"] = 1e-3
        if rng.random() < 0.2:
            c["gravity"] = 0.1
    return c


# ---- meshes and initial states ------------------------------------------------------------------
_meshes = {}


def _settings(c):
    return MHDSettings(gamma0=1.4 if c["problem"] == "kh" else 5.0 / 3.0, cfl=0.4, slope_type=c["slope_type"],
                       riemann="HLLD", time_integrator=c["integrator"],
                       gravity=(0.0, -c["gravity"], 0.0) if c["gravity"] else None,
                       viscosity_mu=c["mu"] if c["mu"] else None)


def _loop_levels(c):
    """Refinement levels of the batch's problems: cell counts log-uniform between 32 and 256 cells in y."""
    rng = random.Random(1000 + c["problems"])
    return [rng.randint(1, 4) for _ in range(c["problems"])]


def _mesh(c):
    """(mesh, problem ids or None). The mesh is a plain function of the case: kept for its next preparation."""
    key = tuple(c[k] for k in ("problem", "dim", "level", "max_level", "bricks", "block", "walls", "problems"))
    if key not in _meshes:
        b, dim = c["block"], c["dim"]
        block = (b, b, b if dim == 3 else 1)
        if c["problem"] == "loops":
            made = BlockMesh.batch([BlockMesh.uniform(2, bricks=(2, 1, 1), level=lv, block=block) for lv in _loop_levels(c)])
        elif c["max_level"]:
            if c["problem"] == "kh":
                def refine(level, lo, hi):
                    return any(lo[1] - 0.02 <= yl <= hi[1] + 0.02 for yl in (0.25, 0.75))
            else:
                refine = workloads.refine_band((0.5, 0.5, 0.5), 0.08, 0.12)
            made = (BlockMesh.amr(dim, refine, base_level=c["level"], max_level=c["max_level"], block=block,
                                  periodic=(True, not c["walls"], True)), None)
        else:
            made = (BlockMesh.uniform(dim, bricks=(c["bricks"], 1, 1), level=c["level"], block=block), None)
        _meshes.clear()
        _meshes[key] = made
    return _meshes[key]


def _lengths(c):
    """Extent of the domain along x, y, z (one root tree has unit length)."""
    return (2.0 if c["problem"] == "loops" else float(c["bricks"]), 1.0, 1.0)


def _state(c, mesh, seed, device):
    """U, B of the case's problem: cell averages from the problem's fields with seeded amplitudes and phases, face
    B as the discrete curl of A_z at the edges (divergence-free, equal on both copies of a shared face)."""
    rng = np.random.default_rng(seed)
    bx, by, bz = mesh.block
    n, dim, gamma = mesh.n_blocks, mesh.dim, _settings(c).gamma0
    Lx, Ly, Lz = _lengths(c)
    two = 2.0 * math.pi
    f8 = dict(dtype=torch.float64, device=device)
    dx = torch.from_numpy(mesh.block_dx()).to(device)[:, None, None, None]
    co = torch.from_numpy(mesh.coords).to(device)
    org = [co[:, d, None, None, None].double() for d in range(3)]

    def pos(axis, count, centre, wrap):
        shape = [1, 1, 1, 1]
        shape[3 - axis] = count
        g = org[axis] * mesh.block[axis] + torch.arange(count, **f8).reshape(shape)
        L = (Lx, Ly, Lz)[axis]
        if wrap and mesh.periodic[axis]:
            g = torch.remainder(g, torch.round(L / dx))
        return (g + (0.5 if centre else 0.0)) * dx

    xc, yc, zc = pos(0, bx, True, False), pos(1, by, True, False), pos(2, bz, True, False)
    if dim == 2:
        zc = torch.zeros_like(zc)
    U = torch.zeros((n, 5, bz, by, bx), **f8)
    B = torch.zeros((n, mesh.nface), **f8)
    nfx, nfy, _ = mesh.face_counts
    Bx = B[:, :nfx].reshape(n, bz, by, bx + 1)
    By = B[:, nfx:nfx + nfy].reshape(n, bz, by + 1, bx)
    Bz = B[:, nfx + nfy:].reshape(n, bz + (dim == 3), by, bx)
    noise = torch.Generator(device=device).manual_seed(seed)
    shape = (n, bz, by, bx)
    one = torch.ones(shape, **f8)
    if c["problem"] == "ot":
        a1, a2 = rng.uniform(0.8, 1.2, 2)
        p1, p2, p3 = rng.uniform(0.0, two, 3)
        b0 = 1.0 / math.sqrt(4.0 * math.pi)

        def az(x, y, z):
            f = b0 * (a1 * torch.cos(2 * two * x / Lx + p1) / (2 * two) + a2 * torch.cos(two * y + p2) / two)
            return f * (1.0 + 0.2 * torch.sin(two * z + p3)) if dim == 3 else f

        rho = 25.0 / (36.0 * math.pi) * (1.0 + 1e-3 * (2.0 * torch.rand(shape, generator=noise, **f8) - 1.0))
        p = 5.0 / (12.0 * math.pi) * one
        vx, vy = -torch.sin(two * yc + p2) * one, torch.sin(two * xc / Lx + p1) * one
        vz = 0.2 * torch.sin(two * zc + p3) * one
        bz0 = 0.1
    elif c["problem"] == "blast":
        r0, pin, ang = 0.1, rng.uniform(8.0, 12.0), rng.uniform(0.6, 0.9)
        bx0, by0 = math.cos(ang), math.sin(ang)

        def az(x, y, z):
            return 0.0 * x * y
        r = torch.sqrt((xc - 0.5) ** 2 + (yc - 0.5) ** 2 + ((zc - 0.5) ** 2 if dim == 3 else 0.0 * zc))
        rho = 1.0 + 1e-3 * (2.0 * torch.rand(shape, generator=noise, **f8) - 1.0)
        vx, vy, vz = 0.0 * one, 0.0 * one, 0.0 * one
        p = torch.where(r < r0, pin, 0.1) * one
        bz0 = 0.0
    elif c["problem"] == "kh":
        amp, ph = rng.uniform(0.008, 0.012), rng.uniform(0.0, two)

        def az(x, y, z):
            return 0.0 * x * y
        s = 0.5 * (1.0 + torch.tanh((0.25 - torch.abs(yc - 0.5)) / 0.01)) * one
        rho, vx, p = 1.0 + s, -0.5 + s, 2.5 * one
        vy = amp * torch.sin(2 * two * xc + ph) + 1e-3 * torch.randn(shape, generator=noise, **f8)
        vz, bz0 = 0.0 * one, 0.0
    else:
        per = torch.from_numpy(rng.uniform(0.0, 1.0, (c["problems"], 3))).to(device)
        per = per[torch.from_numpy(_mesh(c)[1]).to(device).long()][:, :, None, None, None]
        rad, speed, ang = 0.2 + 0.15 * per[:, 0], 1.0 + 2.0 * per[:, 1], two * per[:, 2]

        def az(x, y, z):
            return 1e-3 * torch.clamp(rad - torch.sqrt((x - 1.0) ** 2 + (y - 0.5) ** 2), min=0.0)
        rho, p, vz, bz0 = one, one, 0.0 * one, 0.0
        vx, vy = speed * torch.cos(ang) * one, speed * torch.sin(ang) * one
    Bz += bz0
    if c["problem"] == "blast":
        Bx += bx0
        By += by0
    elif c["problem"] == "kh":
        Bx += 0.1
    else:
        xe, ye = pos(0, bx + 1, False, True), pos(1, by + 1, False, True)
        a = az(xe, ye, zc)
        Bx += (a[:, :, 1:, :] - a[:, :, :-1, :]) / dx
        By -= (a[..., 1:] - a[..., :-1]) / dx
        del a
    bcx, bcy = 0.5 * (Bx[..., 1:] + Bx[..., :-1]), 0.5 * (By[:, :, 1:] + By[:, :, :-1])
    bcz = 0.5 * (Bz[:, 1:] + Bz[:, :-1]) if dim == 3 else Bz
    U[:, 0], U[:, 2], U[:, 3], U[:, 4] = rho, rho * vx, rho * vy, rho * vz
    U[:, 1] = p / (gamma - 1.0) + 0.5 * rho * (vx * vx + vy * vy + vz * vz) + 0.5 * (bcx ** 2 + bcy ** 2 + bcz ** 2)
    if mesh.n_blocks > mesh.n_owned:  # outside blocks: filled by the solver before each step
        U[mesh.n_owned:] = 0.0
        B[mesh.n_owned:] = 0.0
    return U, B


def _dt(c, mesh, U, B):
    """A time step within the CFL limit, from a bound on the fastest speed (a plain power-of-two fraction of dx)."""
    n = mesh.n_owned
    dx = float(mesh.block_dx()[:n].min())
    rho = U[:n, 0]
    p = (_settings(c).gamma0 - 1.0) * float((U[:n, 1] / rho).max())
    v = max(float((U[:n, d].abs() / rho).max()) for d in (2, 3, 4))
    a = float(B[:n].abs().max()) / math.sqrt(float(rho.min()))
    limit = 0.4 * dx / (c["dim"] * (math.sqrt(_settings(c).gamma0 * p + 2.0 * a * a) + v))
    return 2.0 ** math.floor(math.log2(limit))


def prepare(case, seed):
    c = {**DEFAULTS, **case}
    mesh, problem = _mesh(c)
    U, B = _state(c, mesh, seed, "cuda")
    kw = dict(problem=problem, n_problems=c["problems"]) if problem is not None else {}
    if c["walls"]:
        kw["bc"] = (1, 1, 3, 3, 1, 1)
    impl = GodunovImplemGB300(_settings(c), mesh, precision=c["precision"], **kw)
    s = {"c": c, "mesh": mesh, "impl": impl, "U": U, "B": B}
    if c["call"] == "host":
        s["dt"] = _dt(c, mesh, U, B)
        host = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True) for t in (U, B, U, B)]
        host[0].copy_(U)
        host[1].copy_(B)
        s["keep"] = host
        s["host"] = [t.numpy() for t in host]
        del s["U"], s["B"]
    elif c["call"] in ("step", "advance"):
        s["U2"], s["B2"] = torch.zeros_like(U), torch.zeros_like(B)
        if c["call"] == "step":
            s["dt"] = _dt(c, mesh, U, B)
        else:
            s["Uw"], s["Bw"] = torch.empty_like(U), torch.empty_like(B)
    return s


def run(s):
    c, impl = s["c"], s["impl"]
    if c["call"] == "step":
        if c["walls"]:
            impl.fill_outside(s["U"], s["B"])
        impl.do_time_step(s["U"], s["U2"], s["B"], s["B2"], s["dt"])
        return {"U": s["U2"], "B": s["B2"]}
    if c["call"] == "inv_dt":
        return {"inv_dt": impl.compute_inv_dt(s["U"], s["B"])}
    if c["call"] == "host":
        U, B, U2, B2 = s["host"]
        impl.step_host(U, B, s["dt"], U2, B2)
        return {"U": U2, "B": B2}
    if c["call"] == "advance":
        s["Uw"].copy_(s["U"])
        s["Bw"].copy_(s["B"])
        dt_log, t = impl.advance(s["Uw"], s["U2"], s["Bw"], s["B2"], c["steps"])
        return {"U": s["Uw"], "B": s["Bw"], "dt": dt_log, "t": t}
    impl.resize_auxiliary_data(s["mesh"])
    mesh, U, B = impl.regrid(s["U"], s["B"], c["level"], c["max_level"], criterion="SIMPLE_GRADIENT", eps_refine=0.1,
                             eps_coarsen=0.05, variables=("rho", "pressure"))
    return {"U": U, "B": B, "level": mesh.level, "flags": impl.last_flags}


def work(case):
    """Bytes: U (5 values a cell) and face B read and written once in FP64. Operations: the scheme's own, once a
    cell, counted from its formulas (slopes, predictor, edge field, face fluxes, edge EMFs, update)."""
    c = {**DEFAULTS, **case}
    mesh = _mesh(c)[0]
    state = 8.0 * mesh.n_owned * (5 * mesh.ncell + mesh.nface)
    cells = float(mesh.n_owned * mesh.ncell)
    if c["call"] == "inv_dt":
        return {"bytes": state, "flops": 60.0 * cells}
    if c["call"] == "regrid":
        return {"bytes": 2.0 * state, "flops": 50.0 * cells}
    stages = c["steps"] * (2 if c["integrator"] == "RK2_SSP" else 1) if c["call"] == "advance" else 1
    per = 2600.0 if c["dim"] == 3 else 1100.0
    return {"bytes": 2.0 * state * stages, "flops": per * cells * stages}


# ---- the same in plain torch, 64 bits, on arrays over the whole (periodic) domain ---------------
def _gather(c, mesh, U, B):
    """[([5, P, z, y, x], [Bx, By, Bz], block ids)] of groups of equal problems; faces: those at each cell's left."""
    bx, by, bz = mesh.block
    nfx, nfy, _ = mesh.face_counts
    levels = _loop_levels(c) if c["problem"] == "loops" else [c["level"]]
    prob = _mesh(c)[1] if c["problem"] == "loops" else np.zeros(mesh.n_owned, np.int32)
    out = []
    for lv in sorted(set(levels)):
        members = [i for i, v in enumerate(levels) if v == lv]
        ids = np.concatenate([np.nonzero(prob == m)[0] for m in members])
        P = len(members)
        co = torch.from_numpy(mesh.coords[ids]).to(U.device)
        g = [int(co[:, d].max()) + 1 for d in range(3)]
        at = (torch.arange(P, device=U.device).repeat_interleave(len(ids) // P), co[:, 2], co[:, 1], co[:, 0])
        sel = torch.from_numpy(ids).to(U.device)

        def whole(blocks, at=at, P=P, g=g):
            w = torch.empty((P, g[2], g[1], g[0], bz, by, bx), dtype=torch.float64, device=blocks.device)
            w[at] = blocks
            return w.permute(0, 1, 4, 2, 5, 3, 6).reshape(P, g[2] * bz, g[1] * by, g[0] * bx)

        Ub, Bb = U[sel], B[sel]
        faces = [whole(Bb[:, :nfx].reshape(-1, bz, by, bx + 1)[..., :-1]),
                 whole(Bb[:, nfx:nfx + nfy].reshape(-1, bz, by + 1, bx)[:, :, :-1]),
                 whole(Bb[:, nfx + nfy:].reshape(-1, bz + (mesh.dim == 3), by, bx)[:, :bz])]
        dx = 1.0 / float(mesh.block[0] << lv)
        out.append({"U": [whole(Ub[:, v]) for v in range(5)], "F": faces, "dx": dx, "sel": sel, "at": at, "g": g,
                    "members": members})
    return out


def _scatter(mesh, groups, U, B):
    """The groups' arrays back into the blocks' layout (both copies of a shared face)."""
    bx, by, bz = mesh.block
    nfx, nfy, _ = mesh.face_counts
    for q in groups:
        g, at, P = q["g"], q["at"], len(q["members"])

        def blocks(w, axis=None):
            def cut(a):
                return a.reshape(P, g[2], bz, g[1], by, g[0], bx).permute(0, 1, 3, 5, 2, 4, 6)[at]
            if axis is None:
                return cut(w)
            last = cut(torch.roll(w, -1, axis)).narrow(axis, (bx, by, bz)[-1 - axis] - 1, 1)
            return torch.cat([cut(w), last], axis)

        for v in range(5):
            U[q["sel"], v] = blocks(q["U"][v])
        parts = [blocks(q["F"][0], -1), blocks(q["F"][1], -2), blocks(q["F"][2], -3 if mesh.dim == 3 else None)]
        B[q["sel"]] = torch.cat([p.reshape(len(q["sel"]), -1) for p in parts], 1)


def _sh(a, d, n):
    """Value at index + n along axis d (0: x)."""
    return torch.roll(a, -n, -1 - d) if n else a


def _primitives(st, q, dim):
    Bc = [0.5 * (q["F"][d] + _sh(q["F"][d], d, 1)) for d in range(dim)]
    if dim == 2:
        Bc.append(q["F"][2])
    U = q["U"]
    r = torch.clamp(U[0], min=st.smallr)
    v = [U[2 + d] / r for d in range(3)]
    eint = (U[1] - 0.5 * (Bc[0] ** 2 + Bc[1] ** 2 + Bc[2] ** 2)) / r - 0.5 * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    p = torch.maximum((st.gamma0 - 1.0) * r * eint, r * st.smallp)
    return [r, p] + v, Bc


def _fast(st, d, p, b, bn):
    b2 = b[0] * b[0] + b[1] * b[1] + b[2] * b[2]
    c2 = st.gamma0 * p / d
    h = 0.5 * (b2 / d + c2)
    return torch.sqrt(h + torch.sqrt(torch.clamp(h * h - c2 * bn * bn / d, min=0.0)))


def _inv_dt(st, q, dim):
    Q, Bc = _primitives(st, q, dim)
    s = [_fast(st, Q[0], Q[1], Bc, Bc[d]) + Q[2 + d].abs() for d in range(dim)]
    val = sum(x / q["dx"] for x in s)
    if st.gravity is not None:
        k = sum(abs(g) for g in st.gravity[:dim]) * q["dx"] / sum(x * x for x in s)
        k = torch.clamp(k, min=1e-4)
        val = val * (k / (torch.sqrt(1.0 + 2.0 * k) - 1.0))
    if st.viscosity_mu is not None:
        val = torch.maximum(val, 4.0 * st.viscosity_mu / q["U"][0] / (q["dx"] * q["dx"]))
    return val.amax(dim=(1, 2, 3))


def _slope(q, qp, qm, st):
    a, b, m = st.slope_type * (q - qm), st.slope_type * (qp - q), 0.5 * (qp - qm)
    lim = torch.where(a * b <= 0, torch.zeros_like(a), torch.minimum(a.abs(), b.abs()))
    return torch.where(m >= 0, 1.0, -1.0) * torch.minimum(lim, m.abs())


def _hlld(st, L, R):
    """Miyoshi & Kusano (2005) fluxes; states: rho, p, u, v, w, a, b, c with u, a normal. Returns rho, E, u, v, w, b, c."""
    a = 0.5 * (L[5] + R[5])
    sg = torch.where(a >= 0, 1.0, -1.0)

    def side(q):
        r, p, u, v, w, b, c = q[0], q[1], q[2], q[3], q[4], q[6], q[7]
        em = 0.5 * (a * a + b * b + c * c)
        return p / (st.gamma0 - 1.0) + 0.5 * r * (u * u + v * v + w * w) + em, p + em, u * a + v * b + w * c

    etl, ptl, vbl = side(L)
    etr, ptr, vbr = side(R)
    cf = torch.maximum(_fast(st, L[0], L[1], (a, L[6], L[7]), a), _fast(st, R[0], R[1], (a, R[6], R[7]), a))
    sl, sr = torch.minimum(L[2], R[2]) - cf, torch.maximum(L[2], R[2]) + cf
    rcl, rcr = L[0] * (L[2] - sl), R[0] * (sr - R[2])
    us = (rcr * R[2] + rcl * L[2] + (ptl - ptr)) / (rcr + rcl)
    pts = (rcr * ptl + rcl * ptr + rcl * rcr * (L[2] - R[2])) / (rcr + rcl)

    def star(q, s, et, pt, vb):
        r, u, v, w, b, c = q[0], q[2], q[3], q[4], q[6], q[7]
        rs = r * (s - u) / (s - us)
        e1, e2 = r * (s - u) * (s - us) - a * a, r * (s - u) * (s - u) - a * a
        flat = e1.abs() < 1e-4 * (a * a)
        e1 = torch.where(flat, torch.ones_like(e1), e1)
        vs, bs = torch.where(flat, v, v - a * b * (us - u) / e1), torch.where(flat, b, b * e2 / e1)
        ws, cs = torch.where(flat, w, w - a * c * (us - u) / e1), torch.where(flat, c, c * e2 / e1)
        vbs = us * a + vs * bs + ws * cs
        return rs, vs, ws, bs, cs, vbs, ((s - u) * et - pt * u + pts * us + a * (vb - vbs)) / (s - us), torch.sqrt(rs)

    rsl, vsl, wsl, bsl, csl, vbsl, esl, ql = star(L, sl, etl, ptl, vbl)
    rsr, vsr, wsr, bsr, csr, vbsr, esr, qr = star(R, sr, etr, ptr, vbr)
    sal, sar = us - a.abs() / ql, us + a.abs() / qr
    vss, wss = (ql * vsl + qr * vsr + sg * (bsr - bsl)) / (ql + qr), (ql * wsl + qr * wsr + sg * (csr - csl)) / (ql + qr)
    bss = (ql * bsr + qr * bsl + sg * ql * qr * (vsr - vsl)) / (ql + qr)
    css = (ql * csr + qr * csl + sg * ql * qr * (wsr - wsl)) / (ql + qr)
    vbss = us * a + vss * bss + wss * css
    states = [(rsl, us, vsl, wsl, bsl, csl, pts, esl, vbsl), (rsl, us, vss, wss, bss, css, pts, esl - sg * ql * (vbsl - vbss), vbss),
              (rsr, us, vss, wss, bss, css, pts, esr + sg * qr * (vbsr - vbss), vbss), (rsr, us, vsr, wsr, bsr, csr, pts, esr, vbsr),
              (R[0], R[2], R[3], R[4], R[6], R[7], ptr, etr, vbr)]
    o = (L[0], L[2], L[3], L[4], L[6], L[7], ptl, etl, vbl)
    done = sl > 0
    for state, edge in zip(states, (sal, us, sar, sr, None)):
        o = tuple(torch.where(done, x, y) for x, y in zip(o, state))
        if edge is not None:
            done = done | (edge > 0)
    r, u, v, w, b, c, pt, e, vb = o
    return [r * u, (e + pt) * u - a * vb, r * u * u - a * a + pt, r * u * v - a * b, r * u * w - a * c, b * u - a * v, c * u - a * w]


def _emf(st, RT, LT, RB, LB, perm):
    """2D HLLD EMF at an edge from its four states; perm: positions of (u, v, a, b, c) in the edge's frame."""
    iu, iv, ia, ib, ic = perm
    S = {"LL": RT, "RL": LT, "LR": RB, "RR": LB}
    A = {"LL": 0.5 * (RT[ia] + LT[ia]), "LR": 0.5 * (RB[ia] + LB[ia])}
    A["RL"], A["RR"] = A["LL"], A["LR"]
    Bn = {"LL": 0.5 * (RT[ib] + RB[ib]), "RL": 0.5 * (LT[ib] + LB[ib])}
    Bn["LR"], Bn["RR"] = Bn["LL"], Bn["RL"]
    k4 = ("LL", "RL", "LR", "RR")
    r, p, u, v, C = ({k: S[k][i] for k in k4} for i in (0, 1, iu, iv, ic))
    most = lambda d: torch.stack([d[k] for k in k4]).amax(0)  # noqa: E731
    least = lambda d: torch.stack([d[k] for k in k4]).amin(0)  # noqa: E731
    cx = most({k: _fast(st, r[k], p[k], (A[k], Bn[k], C[k]), A[k]) for k in k4})
    cy = most({k: _fast(st, r[k], p[k], (A[k], Bn[k], C[k]), Bn[k]) for k in k4})
    SL, SR, SB, ST = least(u) - cx, most(u) + cx, least(v) - cy, most(v) + cy
    pt = {k: p[k] + 0.5 * (A[k] ** 2 + Bn[k] ** 2 + C[k] ** 2) for k in k4}
    X = {"LL": SL, "LR": SL, "RL": SR, "RR": SR}
    Y = {"LL": SB, "RL": SB, "LR": ST, "RR": ST}
    rx = {k: r[k] * (u[k] - X[k]).abs() for k in k4}
    ry = {k: r[k] * (v[k] - Y[k]).abs() for k in k4}
    us = (sum(rx[k] * u[k] for k in k4) + (pt["LL"] - pt["RL"] + pt["LR"] - pt["RR"])) / sum(rx.values())
    vs = (sum(ry[k] * v[k] for k in k4) + (pt["LL"] - pt["LR"] + pt["RL"] - pt["RR"])) / sum(ry.values())
    fx = {k: (X[k] - u[k]) / (X[k] - us) for k in k4}
    fy = {k: (Y[k] - v[k]) / (Y[k] - vs) for k in k4}
    As, Bs = {k: A[k] * fy[k] for k in k4}, {k: Bn[k] * fx[k] for k in k4}
    E = {k: u[k] * Bn[k] - v[k] * A[k] for k in k4}
    Ex, Ey = {k: us * Bs[k] - v[k] * A[k] for k in k4}, {k: u[k] * Bn[k] - vs * As[k] for k in k4}
    Es = {k: us * Bs[k] - vs * As[k] for k in k4}
    ax = {k: torch.maximum(A[k].abs() / torch.sqrt(r[k] * fx[k]), As[k].abs() / torch.sqrt(r[k] * fx[k] * fy[k])) for k in k4}
    ay = {k: torch.maximum(Bn[k].abs() / torch.sqrt(r[k] * fy[k]), Bs[k].abs() / torch.sqrt(r[k] * fx[k] * fy[k])) for k in k4}
    two = lambda d, a, b: torch.clamp(torch.maximum(d[a], d[b]), min=st.smallc)  # noqa: E731
    SAL = torch.clamp(us - two(ax, "LR", "LL"), max=0.0)
    SAR = torch.clamp(us + two(ax, "RR", "RL"), min=0.0)
    SAB = torch.clamp(vs - two(ay, "LL", "RL"), max=0.0)
    SAT = torch.clamp(vs + two(ay, "LR", "RR"), min=0.0)
    w, h = SAR - SAL, SAT - SAB
    AT, AB = (SAR * As["RR"] - SAL * As["LR"]) / w, (SAR * As["RL"] - SAL * As["LL"]) / w
    BR, BL = (SAT * Bs["RR"] - SAB * Bs["RL"]) / h, (SAT * Bs["LR"] - SAB * Bs["LL"]) / h
    mid = ((SAL * SAB * Es["RR"] - SAL * SAT * Es["RL"] - SAR * SAB * Es["LR"] + SAR * SAT * Es["LL"]) / w / h
           - SAT * SAB / h * (AT - AB) + SAR * SAL / w * (BR - BL))
    bot = (SAR * Ex["LL"] - SAL * Ex["RL"] + SAR * SAL * (Bn["RL"] - Bn["LL"])) / w
    top = (SAR * Ex["LR"] - SAL * Ex["RR"] + SAR * SAL * (Bn["RR"] - Bn["LR"])) / w
    lef = (SAT * Ey["LL"] - SAB * Ey["LR"] - SAT * SAB * (A["LR"] - A["LL"])) / h
    rig = (SAT * Ey["RL"] - SAB * Ey["RR"] - SAT * SAB * (A["RR"] - A["RL"])) / h

    def across(lo, m, hi):
        return torch.where(SL > 0, lo, torch.where(SR < 0, hi, m))
    return torch.where(SB > 0, across(E["LL"], bot, E["RL"]),
                       torch.where(ST < 0, across(E["LR"], top, E["RR"]), across(lef, mid, rig)))


def _stage(st, q, dim, dt):
    """One MUSCL-Hancock + constrained-transport stage of a periodic problem; dt: per problem."""
    dt = dt.reshape(-1, 1, 1, 1)
    k, F, ax = dt / q["dx"], q["F"], range(dim)
    rk2 = st.time_integrator == "RK2_SSP"
    Q, Bc = _primitives(st, q, dim)
    r, p, u, v, w = Q
    A, B, C = Bc
    zero = torch.zeros_like(r)
    S = []
    for d in ax:
        s = [_slope(x, _sh(x, d, 1), _sh(x, d, -1), st) for x in Q[:5 if dim == 3 else 4]]
        s += [zero] * (5 - len(s))
        for m in range(3):
            s.append(_sh(F[m], m, 1) - F[m] if m == d else _slope(Bc[m], _sh(Bc[m], d, 1), _sh(Bc[m], d, -1), st))
        S.append(s)
    if rk2:
        W = Q + Bc
    else:
        sr, sp = zero, zero
        sv, sb = [zero] * 3, [zero] * 3
        V = Q[2:]
        for d in ax:
            D = S[d]
            sr = sr + (-V[d] * D[0] - D[2 + d] * r) * k
            sp = sp + (-V[d] * D[1] - D[2 + d] * st.gamma0 * p) * k
            grad = D[1] + sum(Bc[m] * D[5 + m] for m in range(3) if m != d)
            sv = [sv[m] + (-V[d] * D[2 + m] - (grad if m == d else -Bc[d] * D[5 + m]) / r) * k for m in range(3)]
            # the face-normal field's own gradient stays out of the tension term of the normal velocity
            sb = [sb[m] if m == d else
                  sb[m] + (V[m] * D[5 + d] + Bc[d] * D[2 + m] - V[d] * D[5 + m] - Bc[m] * D[2 + d]) * k for m in range(3)]
        g = [x for x in (st.gravity or (0.0, 0.0, 0.0))]
        W = [r + 0.5 * sr, p + 0.5 * sp]
        W += [V[m] + (0.5 * dt * g[m] if m < dim else 0.0) + 0.5 * sv[m] for m in range(3)]
        W += [Bc[m] + 0.5 * sb[m] for m in range(3)]

    def edge_avg(x, d0, d1):
        return 0.25 * (x + _sh(x, d0, -1) + _sh(x, d1, -1) + _sh(_sh(x, d0, -1), d1, -1))

    def edge_e(d0, d1):
        return (edge_avg(Q[2 + d0], d0, d1) * 0.5 * (F[d1] + _sh(F[d1], d0, -1))
                - edge_avg(Q[2 + d1], d0, d1) * 0.5 * (F[d0] + _sh(F[d0], d1, -1)))
    Ez = edge_e(0, 1)
    up = lambda e, d: (_sh(e, d, 1) - e) * 0.5 * k  # noqa: E731
    if dim == 3:
        Ex, Ey = edge_e(1, 2), edge_e(2, 0)
        H = [up(Ez, 1) - up(Ey, 2), up(Ex, 2) - up(Ez, 0), up(Ey, 0) - up(Ex, 1)]
    else:
        H = [up(Ez, 1), -up(Ez, 0)]

    floor = lambda q8: [torch.clamp(q8[0], min=st.smallr)] + [  # noqa: E731
        torch.maximum(st.smallp * torch.clamp(q8[0], min=st.smallr), q8[1])] + q8[2:]
    U = q["U"] + ([F[2]] if dim == 2 else [])
    new = list(U)
    for d in ax:
        L = floor([_sh(W[n] + 0.5 * S[d][n], d, -1) for n in range(8)])
        R = floor([W[n] - 0.5 * S[d][n] for n in range(8)])
        L[5 + d] = R[5 + d] = F[d] + H[d]
        order = [0, 1, 2, 3, 4, 5, 6, 7]
        order[2], order[2 + d], order[5], order[5 + d] = 2 + d, 2, 5 + d, 5
        f = _hlld(st, [L[n] for n in order], [R[n] for n in order])
        f = f[:5] + [zero] + f[5:]
        f = [f[n] for n in order]
        for n in range(len(U)):
            fn = f[n] if n < 5 else f[7]
            new[n] = new[n] + (fn - _sh(fn, d, 1)) * k
        del L, R, f
    if st.viscosity_mu is not None:
        mu, frac = st.viscosity_mu, 0.5 if dim == 2 else 1.0 / 3.0
        G = [[(Q[2 + m] - _sh(Q[2 + m], e, -1)) / q["dx"] for e in ax] for m in ax]
        div = sum(G[m][m] for m in ax)
        for d in ax:
            tau = [2.0 * mu * (G[d][d] - frac * div) if m == d else mu * (G[m][d] + G[d][m]) for m in ax]
            for n, f in [(1, -sum(Q[2 + m] * tau[m] for m in ax))] + [(2 + m, -tau[m]) for m in ax]:
                new[n] = new[n] + (f - _sh(f, d, 1)) * k
    if st.gravity is not None:
        kin = lambda m: 0.5 * sum(m[2 + d] ** 2 for d in ax) / new[0]  # noqa: E731
        before = kin(new)
        for d in ax:
            new[2 + d] = new[2 + d] + dt * st.gravity[d] * (U[0] + new[0]) / 2
        new[1] = new[1] + (kin(new) - before)

    def at_edge(c0, c1, d0, d1, s0, s1):
        """State of the cell at offset (c0, c1) from an edge along the third axis, taken to the edge (side s0, s1 = +-1)."""
        D0, D1 = S[d0], S[d1]
        q8 = [W[n] + 0.5 * (s0 * D0[n] + s1 * D1[n]) for n in range(5)]
        faces = []
        for d, o, s, so in ((d0, d1, s0, s1), (d1, d0, s1, s0)):
            f = F[d]
            val = f if rk2 else f + H[d]
            val = val + 0.5 * so * _slope(f, _sh(f, o, 1), _sh(f, o, -1), st)
            faces.append(_sh(val, d, 1) if s > 0 else val)
        h = [W[5 + m] + 0.5 * (s0 * D0[5 + m] + s1 * D1[5 + m]) for m in range(3)]
        if (d0, d1) == (0, 1):
            # z edges: By is the face's; in 3D Bz takes its slopes once, as the other cell-centred one
            b8 = [faces[0], faces[1], h[2]]
        elif (d0, d1) == (0, 2):
            # y edges: the cell's By takes its slopes twice, as the scheme has it
            b8 = [faces[0], W[6] + (s0 * D0[6] + s1 * D1[6]), faces[1]]
        else:
            # x edges: the y face's value, and the cell's By slopes on top of it, as the scheme has it
            b8 = [h[0], faces[0] + 0.5 * (s0 * D0[6] + s1 * D1[6]), faces[1]]
        q8 = floor(q8 + b8)
        return [_sh(_sh(x, d0, c0), d1, c1) for x in q8]

    def emf(d0, d1, perm, swap):
        LB, RT = at_edge(0, 0, d0, d1, -1, -1), at_edge(-1, -1, d0, d1, 1, 1)
        RB, LT = at_edge(-1, 0, d0, d1, 1, -1), at_edge(0, -1, d0, d1, -1, 1)
        if swap:
            RB, LT = LT, RB
        return _emf(st, RT, LT, RB, LB, perm) * k
    Mz = emf(0, 1, (2, 3, 5, 6, 7), False)
    df = lambda e, d: _sh(e, d, 1) - e  # noqa: E731
    if dim == 3:
        My, Mx = emf(0, 2, (4, 2, 7, 5, 6), True), emf(1, 2, (3, 4, 6, 7, 5), False)
        faces = [F[0] + df(Mz, 1) - df(My, 2), F[1] + df(Mx, 2) - df(Mz, 0), F[2] + df(My, 0) - df(Mx, 1)]
    else:
        faces = [F[0] + df(Mz, 1), F[1] - df(Mz, 0), new[5]]
    return {**q, "U": new[:5], "F": faces}


def exact(case, seed):
    """The stage in 64 bits on uniform periodic meshes. Coarse/fine meshes and walls have no such plain form (their
    ghost values are defined by the package's own prolongation), nor has the regridded state."""
    c = {**DEFAULTS, **case}
    if c["max_level"] or c["walls"] or c["call"] == "regrid":
        return None
    st = _settings(c)
    mesh = _mesh(c)[0]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    U, B = _state(c, mesh, seed, device)
    dim, groups = c["dim"], _gather(c, mesh, U, B)
    if c["call"] == "inv_dt":
        return {"inv_dt": float(max(_inv_dt(st, q, dim).max() for q in groups))}
    if c["call"] in ("step", "host"):
        dt = torch.tensor([_dt(c, mesh, U, B)], dtype=torch.float64, device=device)
        _scatter(mesh, [_stage(st, q, dim, dt) for q in groups], U, B)
        return {"U": U, "B": B} if c["call"] == "step" else {"U": U.cpu().numpy(), "B": B.cpu().numpy()}
    dts = np.zeros((c["steps"], c["problems"]))
    for n in range(c["steps"]):
        for i, q in enumerate(groups):
            dt = st.cfl / _inv_dt(st, q, dim)
            dts[n, q["members"]] = dt.cpu().numpy()
            s = _stage(st, q, dim, dt)
            if c["integrator"] == "RK2_SSP":
                s = _stage(st, s, dim, dt)
                s["U"] = [0.5 * a + 0.5 * b for a, b in zip(q["U"], s["U"])]
                s["F"] = [0.5 * a + 0.5 * b for a, b in zip(q["F"], s["F"])]
            groups[i] = s
    _scatter(mesh, groups, U, B)
    return {"U": U, "B": B, "dt": dts, "t": dts.sum(0)}
