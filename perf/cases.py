"""Performance cases of the FLIP step, each through the public entry points.

A case is a plain dict.  "kind" names the call that a program makes:

  step      fsim_step_host: one whole step of a particle state that lives in
            pinned host memory, as the reference's runtime keeps it (upload,
            move and rebin, P2G, pressure solve, G2P, download).
  project   the per-stage calls of FlipDriver::RunOneStep between the move
            and G2P on a device-resident state (the drop-in path of programs
            written against FlipSimulation): P2G, boundary conditions, saved
            velocities, gravity, divergence, fp32 pressure solve, projection;
            the projected face velocities and the pressure come back.
  solve     fsim_pcg_solve alone on an assembled system, in each precision;
            the pressure comes back.
  gradient  a differentiable one-step rollout, forward and backward, as a
            control loop takes it; the gradients go to fp32 parameters.
  levelset  particles to a level set, as the converter for rendered frames
            does once per frame.

Scenes are the synthetic ones of the benchmark and the tests (sphere drop,
dam break, multi-dam), scaled to the case's dimensions, with seeded particle
positions.  Velocities are a vortical flow with noise, so that fields are far
from rest, at the time step 1/300 s that the driver's rule gives fast flows.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("fluid-sim-lb_gb300"))
import fsim  # noqa: E402

DT = 1.0 / 300.0
FLIP = 0.95
TOL = {"fp32": 1e-5, "mixed": 1e-6, "fp64": 1e-8}
PREC = {"fp32": fsim.PREC_FP32, "mixed": fsim.PREC_MIXED, "fp64": fsim.PREC_FP64}
# share of the domain's cells that hold fluid, and PCG iterations to 1e-5 per
# cell of the domain's height (measured on the benchmark's scenes)
FILL = {"sphere_drop": 0.214, "dam_break": 0.24, "multidam": 0.122}
ITERS = {"sphere_drop": 1.5, "dam_break": 2.6, "multidam": 1.3}


def _case(name, kind, scene, nx, ny, nz, prec="fp32", ppc=8, tank=False, block=False):
    return {"name": name, "kind": kind, "scene": scene, "nx": nx, "ny": ny, "nz": nz,
            "prec": prec, "ppc": ppc, "tank": tank, "block": block}


def listed():
    return [
        # a small interactive scene: launches and latency decide
        _case("step_32", "step", "sphere_drop", 32, 32, 32),
        # the benchmark's 64^3 configuration from host memory
        _case("step_64", "step", "sphere_drop", 64, 64, 64),
        # an odd-sized tank with a solid block, fewer particles per cell
        _case("step_ragged", "step", "dam_break", 121, 77, 94, ppc=6, tank=True, block=True),
        # the headline configuration, end to end
        _case("step_256", "step", "dam_break", 256, 256, 256),
        # the stage calls on mid-sized and headline-sized device states
        _case("project_128", "project", "sphere_drop", 128, 128, 128),
        _case("project_256", "project", "dam_break", 256, 256, 256),
        # one-off solves: double precision (reference gradients, checks) ...
        _case("solve_fp64_96", "solve", "sphere_drop", 96, 96, 96, prec="fp64"),
        # ... the mixed-precision solver at a size that fits on chip ...
        _case("solve_mixed_128", "solve", "sphere_drop", 128, 128, 128, prec="mixed"),
        # ... and both fast solvers on the 512^3 multi-dam (16.4 M unknowns)
        _case("solve_fp32_512", "solve", "multidam", 512, 512, 512),
        _case("solve_mixed_512", "solve", "multidam", 512, 512, 512, prec="mixed"),
        # gradients of a small control problem
        _case("gradient_48", "gradient", "sphere_drop", 48, 48, 48, prec="mixed"),
        # a frame's surface for rendering
        _case("levelset_128", "levelset", "sphere_drop", 128, 128, 128),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "project", "project", "solve", "solve", "gradient",
                       "levelset"])
    prec, ppc, tank, block = "fp32", 8, False, False
    if kind == "step":
        lo, hi = 24, 210
        ppc = rng.choice([8, 8, 8, 4, 6])
        tank = rng.random() < 0.25
        block = rng.random() < 0.25
    elif kind == "project":
        lo, hi = 24, 210
        ppc = rng.choice([8, 8, 8, 4, 6])
        block = rng.random() < 0.25
    elif kind == "solve":
        prec = rng.choice(["fp32", "mixed", "fp64"])
        lo, hi = 24, {"fp32": 400, "mixed": 400, "fp64": 110}[prec]
    elif kind == "gradient":
        prec, lo, hi = rng.choice(["mixed", "fp64"]), 16, 56
    else:
        lo, hi = 24, 140
    base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    scene = rng.choice(["sphere_drop", "dam_break", "multidam"])
    if base > 260:
        scene = "multidam"
    n = [max(16, int(round(base * rng.uniform(0.8, 1.2)))) for _ in range(3)]
    if kind == "gradient":
        scene = "sphere_drop"
    c = _case("", kind, scene, n[0], n[1], n[2], prec, ppc, tank, block)
    del c["name"]
    return c


def _dims(c):
    return c["nx"], c["ny"], c["nz"]


def _passes(c):
    """The benchmark's scene scaled to the case's dimensions."""
    nx, ny, nz = (float(d) for d in _dims(c))
    if c["scene"] == "sphere_drop":
        return [fsim.SeedPass([
            fsim.SceneShape(fsim.SHAPE_POOL, a=(0.0, 0.2 * ny, 0.0)),
            fsim.SceneShape(fsim.SHAPE_SPHERE, a=(0.5 * nx, 0.7 * ny, 0.5 * nz),
                            r=0.15 * min(nx, ny, nz))])]
    if c["scene"] == "dam_break":
        return [fsim.SeedPass([fsim.SceneShape(fsim.SHAPE_CUBOID, a=(0.0, 0.0, 0.0),
                                               b=(0.4 * nx, 0.6 * ny, nz))])]
    shapes = [fsim.SceneShape(fsim.SHAPE_POOL, a=(0.0, 0.05 * ny, 0.0))]
    for x0 in (0.0, 0.8):
        for z0 in (0.0, 0.8):
            shapes.append(fsim.SceneShape(fsim.SHAPE_CUBOID, a=(x0 * nx, 0.0, z0 * nz),
                                          b=((x0 + 0.2) * nx, 0.5 * ny, (z0 + 0.2) * nz)))
    return [fsim.SeedPass(shapes)]


def _block(c):
    """The solid block of the cases that have one: inclusive cell box."""
    nx, ny, nz = _dims(c)
    return (nx // 5, 0, nz // 3), (nx // 5 + nx // 10, ny // 8, nz // 3 + nz // 5)


def _sim(c):
    g, force = fsim.physical_gravity(c["ny"])
    sim = fsim.Simulation(_dims(c), fsim.BOUNDARY_TANK if c["tank"] else fsim.BOUNDARY_BOX, g,
                          force, FLIP, c["ppc"])
    if c["block"]:
        sim.add_solid_cuboid(*_block(c))
    sim.seed(_passes(c), seed=0)
    return sim


def _pinned(shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _flow(c, pos, gen):
    """Particle velocities: a vortex of about 1 m/s (in a domain 1 m high) whose
    normal component vanishes at the walls, and noise on the FLIP velocity."""
    dims = torch.tensor(_dims(c), dtype=torch.float32, device=pos.device)
    s = pos / dims * math.pi
    a = float(c["ny"]) * (0.75 + 0.5 * torch.rand(3, generator=gen, device=pos.device))
    sn, cs = torch.sin(s), torch.cos(s)
    v = torch.stack([a[0] * sn[:, 0] * cs[:, 1], -a[1] * cs[:, 0] * sn[:, 1],
                     0.2 * a[2] * sn[:, 2] * torch.sin(2.0 * s[:, 0])], 1)
    noise = torch.randn(pos.shape, generator=gen, device=pos.device)
    return v + 0.02 * c["ny"] * noise, v


def _particles(c, seed):
    """The case's initial particles on the device (positions, velocities, PIC
    velocities), and the simulation that seeded them: the scene's cells and
    particle counts, each particle at a seeded place in its cell."""
    sim = _sim(c)
    n = sim.particle_count()
    pos = _pinned((n, 3))
    got = ctypes.c_int64()
    sim._ck(sim.lib.fsim_download_particles(sim.h, pos.data_ptr(), None, None, n,
                                            ctypes.byref(got)), "download_particles")
    pos = pos.cuda().floor_()
    pos = torch.minimum(pos, torch.tensor(_dims(c), device=pos.device) - 1.0)
    gen = torch.Generator(device=pos.device).manual_seed(seed)
    pos += 0.9998 * torch.rand(pos.shape, generator=gen, device=pos.device)
    vel, gvel = _flow(c, pos, gen)
    return sim, pos, vel, gvel


def _params(c):
    p = c["prec"]
    return fsim.pcg_params(fsim.PCG_RELATIVE, PREC[p], 4000, tolerance=TOL[p],
                           inner_tolerance=1e-2, max_refinements=20)


def prepare(case, seed):
    c = case
    dense = tuple(d + 2 for d in _dims(c))
    st = {"kind": c["kind"], "pcg": _params(c)}
    sim, pos, vel, gvel = _particles(c, seed)
    st["sim"] = sim
    host = []
    for t in (pos, vel, gvel):
        h = _pinned(t.shape)
        h.copy_(t)
        host.append(h)
    del pos, vel, gvel
    if c["kind"] == "step":
        st["in"] = host
        # the rows of particles that a step deletes stay zero
        st["out"] = [_pinned(host[0].shape).zero_() for _ in range(3)]
        return st
    sim.upload_particles(*(h.numpy() for h in host))
    if c["kind"] == "solve":
        _assemble(sim)
        st["pressure"] = _pinned(dense)
    elif c["kind"] == "project":
        st["velocity"] = _pinned(dense + (3,))
        st["active"] = _pinned(dense, torch.uint8)
        st["pressure"] = _pinned(dense)
    elif c["kind"] == "gradient":
        st["rollout"] = fsim.Rollout(sim, 1, 1)
        i = np.arange(int(np.prod(dense)) * 3, dtype=np.float64).reshape(dense + (3,))
        st["target"] = (0.1 * c["ny"] * np.sin(1e-3 * i + seed % 1000)).astype(np.float32)
        st["pcg"] = fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_MIXED, 4000, tolerance=1e-9,
                                    inner_tolerance=1e-3, max_refinements=30)
        st["adjoint"] = fsim.pcg_params(fsim.PCG_RELATIVE, PREC[c["prec"]], 4000, tolerance=1e-9,
                                        inner_tolerance=1e-3, max_refinements=30)
    else:
        st["phi"] = _pinned(dense)
        st["active"] = _pinned(dense, torch.uint8)
    return st


def _assemble(sim):
    """RunOneStep's stage calls from P2G to the divergence."""
    sim.clear_grid()
    sim.transfer_particles_to_grid()
    sim.apply_boundary_conditions()
    sim.save_grid_velocities()
    sim.add_gravity(DT)
    sim.apply_boundary_conditions()
    sim.compute_divergence()


def _download(sim, field, out, active=None):
    sim._ck(sim.lib.fsim_download_field(sim.h, field, out.data_ptr(),
                                        None if active is None else active.data_ptr()), "field")


def run(state):
    st, sim = state, state["sim"]
    if st["kind"] == "step":
        _, n = sim.step_host(DT, st["pcg"], *st["in"], out=st["out"])
        return st["out"] + [n]
    if st["kind"] == "project":
        _assemble(sim)
        sim.pcg_solve(st["pcg"])
        sim.update_velocity_from_pressure()
        sim.get_velocity_update()
        _download(sim, fsim.FIELD_VELOCITY, st["velocity"], st["active"])
        _download(sim, fsim.FIELD_PRESSURE, st["pressure"])
        return [st["velocity"], st["pressure"], st["active"]]
    if st["kind"] == "solve":
        sim.pcg_solve(st["pcg"])
        _download(sim, fsim.FIELD_PRESSURE, st["pressure"])
        return [st["pressure"]]
    if st["kind"] == "gradient":
        loss = st["rollout"].forward(DT, st["pcg"], st["target"])
        gv, gg = st["rollout"].backward(st["adjoint"])
        return [loss, gv.astype(np.float32), gg.astype(np.float32)]
    sim._ck(sim.lib.fsim_particles_to_level_set(sim.h, 3.0, 3.0, 1, st["phi"].data_ptr(),
                                                st["active"].data_ptr()), "level_set")
    return [st["phi"], st["active"]]


def work(case):
    c = case
    cells = c["nx"] * c["ny"] * c["nz"]
    dense = (c["nx"] + 2) * (c["ny"] + 2) * (c["nz"] + 2)
    unknowns = FILL[c["scene"]] * cells
    n = unknowns * c["ppc"]
    digits = -math.log10(1e-9 if c["kind"] == "gradient" else TOL[c["prec"]])
    iters = ITERS[c["scene"]] * max(_dims(c)) * digits / 5.0
    # an iteration: the 7-point product (8), p (2), x and r (4), z (1), three dots (6)
    pcg = 21.0 * unknowns * iters
    splat, gather = 3 * 8 * 6.0 * n, 3 * 2 * 21.0 * n
    if c["kind"] == "step":
        return {"bytes": 72.0 * n, "flops": pcg + splat + gather}
    if c["kind"] == "project":
        return {"bytes": 24.0 * n + 17.0 * dense, "flops": pcg + splat}
    if c["kind"] == "solve":
        return {"bytes": (4.0 + 1.0) * unknowns + 4.0 * dense, "flops": pcg}
    if c["kind"] == "gradient":
        return {"bytes": 24.0 * n + 12.0 * dense + 48.0 * n,
                "flops": 2 * pcg + 3 * (splat + gather)}
    band = 4.0 / 3.0 * math.pi * 6.0 ** 3  # voxels within reach of a sphere
    return {"bytes": 12.0 * n + 5.0 * dense, "flops": 9.0 * band * unknowns}


# ---- the same in 64 bits, on dense arrays over the nodes [-1, N + 1] ---------------

def _corner_weights(p, cell, d):
    """The first node of each particle's stencil for component d and its
    offsets from it, per axis."""
    lo, f = [], []
    for ax in range(3):
        b = cell[:, ax]
        if ax != d:
            b = b - (p[:, ax] < b + 0.5).long()
            f.append(p[:, ax] - (b + 0.5))
        else:
            f.append(p[:, ax] - b)
        lo.append(b)
    return lo, f


def _corners(dims, p, cell, d):
    """(node index, weight) of the eight corners, one after the other."""
    lo, f = _corner_weights(p, cell, d)
    for q in range(8):
        o = (q >> 2 & 1, q >> 1 & 1, q & 1)
        w = 1.0
        for ax in range(3):
            w = w * (f[ax] if o[ax] else 1.0 - f[ax])
        i = [lo[ax] + o[ax] + 1 for ax in range(3)]
        yield (i[0] * (dims[1] + 3) + i[1]) * (dims[2] + 3) + i[2], w


def _shifted(a, ax, s):
    """a at the node s (-1 or 1) further along axis ax, zero past the edge."""
    out = torch.zeros_like(a)
    n = a.shape[ax]
    out.narrow(ax, max(0, -s), n - 1).copy_(a.narrow(ax, max(0, s), n - 1))
    return out


def _solid_mask(c, dev):
    n = _dims(c)
    ax = [torch.arange(-1, n[i] + 2, device=dev) for i in range(3)]
    g = torch.meshgrid(*ax, indexing="ij")
    inside = torch.ones_like(g[0], dtype=torch.bool)
    wall = torch.zeros_like(inside)
    for i in range(3):
        inside &= g[i] <= n[i]
        wall |= (g[i] == -1) | (g[i] == n[i])
    s = wall & inside
    if c["block"]:
        lo, hi = _block(c)
        b = torch.ones_like(s)
        for i in range(3):
            b &= (g[i] >= lo[i]) & (g[i] <= min(hi[i], n[i]))
        s |= b
    return s, g


def _solve64(fluid, solid, b):
    """Jacobi-PCG in 64 bits to 1e-13 over the list of fluid cells."""
    dev = b.device
    rows = fluid.reshape(-1).nonzero().squeeze(1)
    m = rows.numel()
    index = torch.full((fluid.numel(),), m, dtype=torch.int32, device=dev)
    index[rows] = torch.arange(m, dtype=torch.int32, device=dev)
    stride = (fluid.shape[1] * fluid.shape[2], fluid.shape[2], 1)
    nbr, diag = [], torch.zeros(m, dtype=torch.float64, device=dev)
    flat = solid.reshape(-1)
    for ax in range(3):
        for s in (-1, 1):
            j = rows + s * stride[ax]
            nbr.append(index[j])
            diag += (~flat[j]).double()
    del index
    rhs = b.reshape(-1)[rows]
    x = torch.zeros_like(rhs)
    r = rhs.clone()
    p = torch.zeros(m + 1, dtype=torch.float64, device=dev)  # its last entry is no cell
    z = r / diag
    p[:m] = z
    rz = torch.dot(r, z)
    stop = 1e-26 * float(torch.dot(rhs, rhs))
    for it in range(12000):
        ap = diag * p[:m]
        for j in nbr:
            ap -= p.index_select(0, j)
        alpha = rz / torch.dot(p[:m], ap)
        x.addcmul_(alpha, p[:m])
        r.addcmul_(-alpha, ap)
        if it % 25 == 0 and float(torch.dot(r, r)) <= stop:
            break
        z = r / diag
        new = torch.dot(r, z)
        p[:m].mul_(new / rz).add_(z)
        rz = new
    out = torch.zeros(fluid.numel(), dtype=torch.float64, device=dev)
    out[rows] = x
    return out.reshape(fluid.shape)


def _grid64(c, pos, vel):
    """P2G to the projected velocity for particles at fp32 positions pos."""
    n = _dims(c)
    shape = tuple(d + 3 for d in n)
    dev = pos.device
    size = shape[0] * shape[1] * shape[2]
    mass = torch.zeros(3, size, dtype=torch.float64, device=dev)
    mom = torch.zeros(3, size, dtype=torch.float64, device=dev)
    on = torch.zeros(size, dtype=torch.bool, device=dev)
    has = torch.zeros(size, dtype=torch.bool, device=dev)
    for i in range(0, pos.shape[0], 1 << 23):
        p = pos[i:i + (1 << 23)].double()
        cell = p.floor().long()
        k = ((cell[:, 0] + 1) * shape[1] + cell[:, 1] + 1) * shape[2] + cell[:, 2] + 1
        has[k] = True
        for d in range(3):
            u = vel[i:i + (1 << 23), d].double()
            for node, w in _corners(n, p, cell, d):
                mass[d].index_add_(0, node, w)
                mom[d].index_add_(0, node, w * u)
                on[node] = True
    on, has = on.reshape(shape), has.reshape(shape)
    u = []
    for d in range(3):
        u.append(torch.where(mass[d] > 1e-5, mom[d] / mass[d], 0.0).reshape(shape))
    del mass, mom
    solid, g = _solid_mask(c, dev)
    fluid = has & ~solid
    for i in range(3):
        fluid &= (g[i] >= 0) & (g[i] < n[i])
    force = fsim.physical_gravity(c["ny"])[1]
    dt = float(np.float32(DT))
    zero = [solid != _shifted(solid, d, -1) for d in range(3)]
    saved = []
    for d in range(3):
        u[d] = torch.where(zero[d], 0.0, u[d])
        saved.append(u[d].clone())
        acc = float(np.float32(np.float32(dt) * np.float32(force[d]))) * (-1.0 if d == 1 else 1.0)
        u[d] = torch.where(on & ~zero[d], u[d] + acc, u[d])
    div = sum(_shifted(u[d], d, 1) - u[d] for d in range(3))
    prs = _solve64(fluid, solid, torch.where(fluid, div, 0.0))
    box = torch.ones_like(on)
    for i in range(3):
        box &= (g[i] >= 0) & (g[i] <= n[i])
    on1 = on.clone()
    for d in range(3):
        low_fluid, low_solid = _shifted(fluid, d, -1), _shifted(solid, d, -1)
        upd = box & ~solid & ~low_solid & (fluid | low_fluid)
        u[d] = torch.where(upd, u[d] + prs - _shifted(prs, d, -1), u[d])
        on1 |= upd
    return u, saved, on, on1, box, prs


def _trim(a):
    return a[:-1, :-1, :-1].contiguous()


def _order(n, cell, live):
    """The live particles by cell in OpenVDB order (64^3 blocks, 8^3 leaves,
    voxels, each x-major), in list order within a cell."""
    key = torch.zeros_like(cell[:, 0])
    for size, count in ((64, [d // 64 + 2 for d in n]), (8, (8, 8, 8)), (1, (8, 8, 8))):
        for ax in range(3):
            key = key * count[ax] + cell[:, ax] // size % (1 << 30 if size == 64 else 8)
    key[~live] = 1 << 62
    return torch.argsort(key, stable=True)[: int(live.sum())]


def _step64(c, pos, vel, gvel):
    n = _dims(c)
    order = _order(n, pos.floor().long(), torch.ones_like(pos[:, 0], dtype=torch.bool))
    pos, vel, gvel = pos[order], vel[order], gvel[order]
    dt = torch.tensor(DT, dtype=torch.float32, device=pos.device)
    pos = pos + gvel * dt  # single precision, as positions are kept
    for d in range(3):
        pos[:, d].clamp_(0.0, float(n[d]))
    cell = pos.floor().long()
    solid, _ = _solid_mask(c, pos.device)
    order = _order(n, cell, ~solid[cell[:, 0] + 1, cell[:, 1] + 1, cell[:, 2] + 1])
    pos, vel, cell = pos[order], vel[order], cell[order]
    u, saved, on0, on1, box, _ = _grid64(c, pos, vel)
    live, total = pos.shape[0], gvel.shape[0]
    new = torch.zeros(total, 3, dtype=torch.float64, device=pos.device)
    pic = torch.zeros_like(new)
    for d in range(3):
        diff = torch.where(box, u[d] - saved[d], saved[d])
        v, diff = torch.where(on1, u[d], 0.0), torch.where(on0, diff, 0.0)
        # the ghost layers -1 and N of the tangential axes take the layer next to them
        a, b = [ax for ax in range(3) if ax != d]

        def ghost(f):
            out = f
            for ax in (a, b):
                i = torch.arange(n[ax] + 3, device=f.device)
                i[0], i[n[ax] + 1] = 1, n[ax]
                out = out.index_select(ax, i)
            # the passes run axis by axis: none reaches the edge at -1 on both
            # axes, and the edge (-1, N) is filled before layer N of axis b is
            for at, src in (((0, 0), (0, 0)), ((0, n[b] + 1), (1, n[b] + 1))):
                to, of = [slice(None)] * 3, [slice(None)] * 3
                to[a], to[b] = at
                of[a], of[b] = src
                out[tuple(to)] = f[tuple(of)]
            return out

        v, diff = ghost(v).reshape(-1), ghost(diff).reshape(-1)
        for i in range(0, live, 1 << 23):
            s = slice(i, min(i + (1 << 23), live))
            vi = di = 0.0
            for node, w in _corners(n, pos[s].double(), cell[s], d):
                vi = vi + w * v[node]
                di = di + w * diff[node]
            pic[s, d] = vi
            new[s, d] = vi + FLIP * (di + vel[s, d].double() - vi)
    return [None, new, pic, None]


def _levelset64(c, pos):
    n = [d + 2 for d in _dims(c)]
    dev = pos.device
    p = pos.double()
    phi = torch.full((n[0] * n[1] * n[2],), 1e9, dtype=torch.float64, device=dev)
    base = p.floor().long()
    lim = torch.tensor(n, device=dev) - 2
    for dx in range(-6, 8):
        for dy in range(-6, 8):
            for dz in range(-6, 8):
                v = base + torch.tensor([dx, dy, dz], device=dev)
                d = (v.double() - p).norm(dim=1) - 3.0
                ok = ((v >= -1) & (v <= lim)).all(1) & (d < 3.0)
                o = ((v[:, 0] + 1) * n[1] + v[:, 1] + 1) * n[2] + v[:, 2] + 1
                phi.scatter_reduce_(0, o[ok], d[ok], "amin")
    phi = phi.clamp_(-3.0, 3.0).reshape(1, 1, *n)
    padded = torch.nn.functional.pad(phi, (1,) * 6, value=3.0)
    mean = torch.nn.functional.avg_pool3d(padded, 3, stride=1)
    return torch.where(phi.abs() < 3.0, mean, phi).clamp_(-3.0, 3.0).reshape(n)


def exact(case, seed):
    c = case
    if c["kind"] == "gradient" or c["tank"]:
        return None
    sim, pos, vel, gvel = _particles(c, seed)
    sim.close()
    if c["kind"] == "step":
        return _step64(c, pos, vel, gvel)
    if c["kind"] == "levelset":
        return [_levelset64(c, pos), None]
    u, _, _, on1, _, prs = _grid64(c, pos, vel)
    if c["kind"] == "solve":
        return [_trim(prs)]
    velocity = torch.stack([_trim(torch.where(on1, f, 0.0)) for f in u], -1)
    return [velocity, _trim(prs), None]
