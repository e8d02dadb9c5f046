"""What the pressure projection is timed on, through its public entry points.

A case names an entry point (``kind``), a scene with its grid, and the
options of the call. Scenes follow ``shiokaze_b200/scenes.py`` (narrow-band
level sets, face velocities held only near the liquid) but are made with
torch on the GPU, from the case and the seed alone. ``exact`` restates each
computation in 64 bits with plain torch operations on dense grids.
"""
from __future__ import annotations

import ctypes
import math
import os

import numpy as np
import torch

from shiokaze_b200 import native
from shiokaze_b200.projection import Grid, MacGrid, MacPressureSolver3
from shiokaze_b200.scenes import PARTICLE_DTYPE

MODEL = os.path.join(os.path.dirname(native.__file__), "models", "shkz_net.bin")
DEV = "cuda"


def listed():
    return [
        # The smallest projection in use: a 64^3 dam break at the default
        # tolerance, inputs resident on the device. Latency and launches.
        dict(name="dambreak_64", kind="project", scene="dambreak", nx=64, ny=64, nz=64, tol=1e-4, dt=0.01),
        # A grid whose sides are multiples of nothing, with moving solids and
        # surface tension: the optional terms and the ragged tiles.
        dict(name="ragged_tension", kind="project", scene="mixed", nx=101, ny=77, nz=90, tol=1e-4, dt=0.005,
             kappa=0.02, moving=True),
        # The everyday projection of a liquid simulation at production size.
        dict(name="tank_256", kind="project", scene="tank", nx=256, ny=256, nz=256, tol=1e-6, dt=0.005),
        # A sparse splash: most tiles of the grid hold no liquid.
        dict(name="splash_384", kind="project", scene="splash", nx=384, ny=384, nz=384, tol=1e-6, dt=0.005),
        # The largest grid: dam break with rain at 512^3.
        dict(name="rain_512", kind="project", scene="rain", nx=512, ny=512, nz=512, tol=1e-6, dt=0.005),
        # The module call of a host simulation: numpy grids in and out.
        dict(name="module_128", kind="module", scene="mixed", nx=128, ny=128, nz=128, tol=1e-4, dt=0.005),
        # The learned preconditioner in the flexible PCG, shipped network.
        dict(name="learned_128", kind="learned", scene="mixed", nx=128, ny=128, nz=128, tol=1e-6, dt=0.005),
        # One application of the network and its weight gradients, as a
        # training step runs them.
        dict(name="network_64", kind="network", scene="mixed", nx=64, ny=64, nz=64, tol=1e-4, dt=0.005),
        # FLIP particles to the grid before a projection: 3-cell band at 8
        # particles a cell, APIC on.
        dict(name="splat_256", kind="splat", scene="tank", nx=256, ny=256, nz=256, per_cell=8, band=3.0, apic=True),
        # Velocity extension after a projection, as the liquid solver asks.
        dict(name="extend_256", kind="extend", scene="tank", nx=256, ny=256, nz=256, width=3),
        # The generic matrix path of LinSolver= with MIC(0).
        dict(name="csr_48", kind="csr", nx=48, ny=48, nz=48, tol=1e-6, mic0=True),
        # The widest full-resolution layer of the network (skip and upsampled
        # input concatenated), without allocation.
        dict(name="conv_128", kind="conv", nx=128, ny=128, nz=128, c0=16, c1=32, cout=16, planes=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["project", "module", "learned", "network", "splat", "extend", "csr", "conv"],
                       [6, 1, 1, 1, 2, 2, 1, 2])[0]
    if kind == "conv":
        c0, c1, cout = rng.choice([(16, 0, 16), (16, 0, 32), (32, 0, 32), (32, 0, 64), (64, 0, 64), (32, 64, 32),
                                   (16, 32, 16)])
        n = [2 * _log(rng, 8, 72) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], c0=c0, c1=c1, cout=cout, planes=8 if cout <= 32 else 4)
    if kind == "csr":
        n = [_log(rng, 12, 48) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], tol=10.0 ** -rng.randint(4, 8), mic0=rng.random() < 0.6)
    top = {"project": 300, "module": 128, "learned": 112, "network": 80, "splat": 256, "extend": 256}[kind]
    base = _log(rng, 32, top)
    n = [max(24, int(base * rng.uniform(0.7, 1.0))) for _ in range(3)]
    scene = rng.choice(["dambreak", "mixed", "tank", "splash", "rain"] if kind == "project" else ["mixed", "tank"])
    case = dict(kind=kind, scene=scene, nx=n[0], ny=n[1], nz=n[2])
    if kind == "splat":
        return dict(case, per_cell=rng.choice([4, 8, 12]), band=rng.choice([2.0, 3.0, 4.0]), apic=rng.random() < 0.8)
    if kind == "extend":
        return dict(case, width=rng.randint(1, 6))
    case.update(tol=10.0 ** -rng.randint(3, 6), dt=rng.choice([0.002, 0.005, 0.01]))
    if kind == "project" and rng.random() < 0.3:
        case.update(kappa=0.02)
    if kind == "project" and rng.random() < 0.3:
        case.update(moving=True)
    if kind == "project" and rng.random() < 0.15:
        case.update(precond="none", tol=1e-3)
    return case


# ----------------------------------------------------------------------
# scenes

def _coords(n, dx, off):
    x, y, z = ((torch.arange(m, device=DEV, dtype=torch.float64) + o) * dx for m, o in zip(n, off))
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _box(x, y, z, lo, hi):
    q = [torch.maximum(lo[a] - c, c - hi[a]) for a, c in enumerate((x, y, z))]
    out = torch.sqrt(sum(v.clamp(min=0) ** 2 for v in q))
    return out + torch.maximum(torch.maximum(q[0], q[1]), q[2]).clamp(max=0)


def _spheres(phi, x, y, z, spheres, dx):
    nz, ny, nx = phi.shape
    for c, r in spheres:
        s = []
        for a, m in enumerate((nx, ny, nz)):
            s.append(slice(max(0, int((c[a] - r) / dx) - 5), min(m, int((c[a] + r) / dx) + 6)))
        if any(t.start >= t.stop for t in s):
            continue
        xs, ys, zs = x[:, :, s[0]], y[:, s[1], :], z[s[2], :, :]
        d = torch.sqrt((xs - c[0]) ** 2 + (ys - c[1]) ** 2 + (zs - c[2]) ** 2) - r
        view = phi[s[2], s[1], s[0]]
        view.copy_(torch.minimum(view, d))
    return phi


class Scene:
    """Device grids of one projection: effective level sets, masks and face
    velocities, [k, j, i] with x fastest; the domain is nx*dx wide, dx = 1/max."""

    def __init__(self, case, seed):
        n = (case["nx"], case["ny"], case["nz"])
        self.n, self.dx = n, 1.0 / max(n)
        dx = self.dx
        L = [m * dx for m in n]
        rs = np.random.RandomState(seed)
        gen = torch.Generator(device=DEV).manual_seed(seed)
        name = case["scene"]

        def balls(count, r0, r1, y0, y1):
            return [([rs.uniform(0.1, 0.9) * L[0], rs.uniform(y0, y1) * L[1], rs.uniform(0.1, 0.9) * L[2]],
                     rs.uniform(r0, r1)) for _ in range(count)]

        def blocks(count, e0, e1):
            got = []
            for _ in range(count):
                c, e = rs.uniform(0.15, 0.85, 3) * L, rs.uniform(e0, e1, 3)
                got.append((c - e / 2, c + e / 2))
            return got

        pool = rs.uniform(0.2, 0.5) * L[1]
        spheres, boxes = [], []
        if name == "dambreak":
            boxes = blocks(1, 0.1, 0.25)
        elif name == "tank":
            boxes = blocks(8, 0.05, 0.2)
        elif name == "splash":
            spheres = balls(200, 0.02, 0.08, 0.4, 0.9)
        elif name == "rain":
            spheres = balls(100, 0.02, 0.06, 0.5, 0.9)
        else:  # "mixed": a pool of random height with spheres and boxes
            spheres = balls(rs.randint(1, 51), 0.02, 0.1, 0.5, 0.9)
            boxes = blocks(rs.randint(1, 9), 0.05, 0.2)

        def fluid(x, y, z):
            full = torch.broadcast_shapes(x.shape, y.shape, z.shape)
            if name == "dambreak":
                phi = torch.minimum(_box(x, y, z, (-1.0, -1.0, -1.0), (0.4 * L[0], 0.6 * L[1], 2.0)),
                                    torch.sqrt((x - 0.5 * L[0]) ** 2 + (y - 0.75 * L[1]) ** 2
                                               + (z - 0.5 * L[2]) ** 2) - 0.15)
            elif name == "tank":
                phi = y - L[1] * (0.5 + 0.1 * torch.sin(2 * math.pi * x / L[0]) * torch.cos(2 * math.pi * z / L[2]))
            elif name == "rain":
                phi = torch.maximum(torch.maximum(x - 0.232 * L[0], y - 0.432 * L[1]),
                                    (z - 0.5 * L[2]).abs() - 0.2532 * L[2])
                phi = torch.minimum(phi, y - 0.095 * L[1])
            else:
                phi = y - (0.3 * L[1] if name == "splash" else pool)
            phi = phi.expand(full).clone()
            return _spheres(phi, x, y, z, spheres, dx)

        def solid(x, y, z):
            out = None
            for lo, hi in boxes:
                v = _box(x, y, z, lo, hi)
                out = v if out is None else torch.minimum(out, v)
            return out

        band = math.sqrt(3.0) * dx

        def push(phi, x, y, z):
            return torch.maximum(phi, -(solid(x, y, z) + dx)) if boxes else phi

        def effective(v):
            v = v.float()
            act = v.double().abs() < band
            return torch.where(act, v, torch.where(v < 0, -band, band).float()), act.to(torch.uint8)

        x, y, z = _coords(n, dx, (0.5, 0.5, 0.5))
        self.phi = push(fluid(x, y, z), x, y, z)  # before banding (particles use it)
        self.fluid, self.fluid_active = effective(self.phi)
        self.solid = self.solid_active = None
        if boxes:
            s = solid(*_coords([m + 1 for m in n], dx, (0.0, 0.0, 0.0))).clamp(max=1.0)
            self.solid, self.solid_active = effective(s)
        self.vel, self.act, self.svel = [], [], None
        for d in range(3):
            shape = [m + (a == d) for a, m in enumerate(n)]
            c = _coords(shape, dx, [0.0 if a == d else 0.5 for a in range(3)])
            on = push(fluid(*c), *c) <= band
            u = torch.empty(shape[::-1], device=DEV)
            if name in ("dambreak", "splash"):
                u.uniform_(-1.0, 1.0, generator=gen)
                u *= 2.0 if name == "splash" else 1.0
            else:
                u.normal_(0.0, 0.5, generator=gen)
            self.vel.append(torch.where(on, u, torch.zeros_like(u)))
            self.act.append(on.to(torch.uint8))
        if case.get("moving"):
            self.svel = [torch.empty_like(v).uniform_(-0.5, 0.5, generator=gen) for v in self.vel]
        if case["kind"] != "splat":
            self.phi = None


def _particles(sc, case, seed):
    """FLIP particle records (uint8 rows on the device) in the liquid's band:
    jittered positions, a smooth velocity with noise, APIC matrices."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 1)
    inside = (sc.fluid < 0) & (sc.phi > -case["band"] * sc.dx)
    cells = inside.nonzero().flip(1).repeat_interleave(case["per_cell"], 0).double()
    p = ((cells + torch.rand(cells.shape, device=DEV, dtype=torch.float64, generator=gen)) * sc.dx).float()
    count = p.shape[0]
    x, y, z = p[:, 0], p[:, 1], p[:, 2]
    v = torch.stack([0.6 * torch.sin(2 * math.pi * y) * torch.cos(math.pi * z),
                     -0.8 * torch.sin(math.pi * x) + 0.3 * torch.cos(2 * math.pi * z),
                     0.4 * torch.cos(2 * math.pi * x) * torch.sin(math.pi * y)], 1)
    v = v + 0.05 * torch.randn(v.shape, device=DEV, generator=gen)
    rec = torch.zeros((count, PARTICLE_DTYPE.itemsize // 4), device=DEV)
    rec[:, 0:3] = p
    rec[:, 3:12] = 2.0 * torch.randn((count, 9), device=DEV, generator=gen)
    rec[:, 12:15] = v
    rec[:, 15] = 0.125 * (0.5 + torch.rand(count, device=DEV, generator=gen))
    rec[:, 16] = 0.25 * sc.dx
    bullet = torch.rand(count, device=DEV, generator=gen) < 0.02
    rec[:, 17].view(torch.int32)[bullet] = 1
    return rec


def _csr(case, seed):
    """A symmetric 7-point system with varying weights (some links absent),
    as compressed rows on the host, and a right-hand side."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rs = np.random.RandomState(seed)
    n = nx * ny * nz
    idx = np.arange(n).reshape(nz, ny, nx)
    rows, cols, vals = [], [], []
    diag = np.zeros(n)
    for axis in (2, 1, 0):
        lo = np.take(idx, range(idx.shape[axis] - 1), axis).ravel()
        hi = np.take(idx, range(1, idx.shape[axis]), axis).ravel()
        keep = rs.rand(lo.size) > 0.02
        lo, hi = lo[keep], hi[keep]
        w = rs.uniform(0.2, 1.0, lo.size)
        np.add.at(diag, lo, w)
        np.add.at(diag, hi, w)
        rows += [lo, hi]
        cols += [hi, lo]
        vals += [-w, -w]
    free = (idx[:, -1, :]).ravel()  # a free surface at the top
    diag[free] += rs.uniform(1.0, 4.0, free.size)
    diag[diag == 0] = 1.0
    rows, cols, vals = (np.concatenate(a + [b]) for a, b in ((rows, np.arange(n)), (cols, np.arange(n)), (vals, diag)))
    order = np.lexsort((cols, rows))
    indptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=indptr[1:])
    return indptr, cols[order].astype(np.int64), vals[order], rs.standard_normal(n)


def _conv_inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    nx, ny, nz, c0, c1, cout = (case[k] for k in ("nx", "ny", "nz", "c0", "c1", "cout"))

    def rnd(*shape):
        return torch.randn(shape, device=DEV, generator=gen)

    in0 = rnd(nz, ny, nx, c0).bfloat16()
    in1 = rnd(nz // 2, ny // 2, nx // 2, c1).bfloat16() if c1 else None
    w = (rnd(27, cout, c0 + c1) / math.sqrt(27 * (c0 + c1))).bfloat16().float()
    return in0, in1, w, 0.1 * rnd(cout)


# ----------------------------------------------------------------------
# the calls

def _ptr(t):
    return None if t is None else t.data_ptr()


def _context(case, **more):
    cfg = native.default_config()
    cfg.residual = case.get("tol", cfg.residual)
    if case.get("precond") == "none":
        cfg.preconditioner = native.PRECOND_NONE
    for k, v in more.items():
        setattr(cfg, k, v)
    return native.Context(cfg)


def _prepare_project(case, sc, ctx):
    nx, ny, nz = sc.n
    st = {"vel": [torch.empty_like(v) for v in sc.vel], "act": [torch.empty_like(m) for m in sc.act],
          "pressure": torch.empty((nz, ny, nx), device=DEV),
          "pressure_active": torch.empty((nz, ny, nx), dtype=torch.uint8, device=DEV), "res": native.Result()}
    a = native.ProjectArgs()
    a.nx, a.ny, a.nz, a.dx, a.dt = nx, ny, nz, sc.dx, case["dt"]
    a.fluid, a.fluid_active = _ptr(sc.fluid), _ptr(sc.fluid_active)
    a.solid, a.solid_active = _ptr(sc.solid), _ptr(sc.solid_active)
    a.pressure, a.pressure_active = _ptr(st["pressure"]), _ptr(st["pressure_active"])
    a.surface_tension = case.get("kappa", 0.0)
    for d in range(3):
        a.velocity[d], a.velocity_active[d] = _ptr(st["vel"][d]), _ptr(st["act"][d])
        if sc.svel is not None:
            a.solid_velocity[d] = _ptr(sc.svel[d])
    st["args"] = a
    return st


def _host_grids(sc):
    np_ = lambda t: t.cpu().numpy()  # noqa: E731
    fluid = Grid(np_(sc.fluid), np_(sc.fluid_active))
    solid = Grid(np_(sc.solid), np_(sc.solid_active)) if sc.solid is not None else None
    return fluid, solid, [np_(v) for v in sc.vel], [np_(m) for m in sc.act]


def _network_inputs(case, seed):
    rs = np.random.RandomState(seed + 7)
    shape = (case["nz"], case["ny"], case["nx"])
    return rs.standard_normal(shape).astype(np.float32), rs


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "conv":
        st["in0"], st["in1"], st["w"], st["b"] = _conv_inputs(case, seed)
        st["out"] = torch.empty((case["nz"], case["ny"], case["nx"], case["cout"]), dtype=torch.bfloat16, device=DEV)
    elif kind == "csr":
        st["indptr"], st["indices"], st["data"], st["b"] = _csr(case, seed)
        st["x"] = np.zeros_like(st["b"])
        st["ctx"] = _context(case, csr_preconditioner=native.PRECOND_MIC0 if case["mic0"] else native.PRECOND_NONE)
        st["res"] = native.Result()
    elif kind in ("module", "network"):
        sc = Scene(case, seed)
        st["solver"] = s = MacPressureSolver3({"Residual": case["tol"]})
        s.initialize(sc.n, sc.dx)
        st["fluid"], st["solid"], st["vel"], st["act"] = _host_grids(sc)
        if kind == "network":
            # the system of a training scene, as a training run has it in hand
            s.project(case["dt"], MacGrid(list(st["vel"]), list(st["act"])), st["solid"], None, st["fluid"])
            s.learned_load(MODEL)
            st["r"], rs = _network_inputs(case, seed)
            nx, ny, nz = s.learned_dims()
            st["g"] = rs.standard_normal((nz, ny, nx)).astype(np.float32)
    else:
        st["sc"] = sc = Scene(case, seed)
        more = {"preconditioner": native.PRECOND_LEARNED} if kind == "learned" else {}
        st["ctx"] = ctx = _context(case, **more)
        if kind == "learned":
            ctx.check(native.load().shkz_b200_learned_load(ctx.handle, MODEL.encode()), "learned_load")
        st["stream"] = torch.cuda.ExternalStream(ctx.stream)
        if kind in ("project", "learned"):
            st.update(_prepare_project(case, sc, ctx))
        else:
            nx, ny, nz = sc.n
            st["vel"], st["act"] = [torch.empty_like(v) for v in sc.vel], [torch.empty_like(m) for m in sc.act]
            if kind == "splat":
                st["rec"] = _particles(sc, case, seed)
                a = native.splat_args(nx, ny, nz, sc.dx, _ptr(st["rec"]), len(st["rec"]), PARTICLE_DTYPE,
                                      apic=case["apic"])
            else:
                a = native.ExtendArgs()
                a.nx, a.ny, a.nz, a.dx, a.width, a.constrain = nx, ny, nz, sc.dx, case["width"], 1
                a.solid, a.solid_active = _ptr(sc.solid), _ptr(sc.solid_active)
            for d in range(3):
                a.velocity[d], a.velocity_active[d] = _ptr(st["vel"][d]), _ptr(st["act"][d])
            st["args"] = a
    torch.cuda.synchronize()
    return st


def run(st):
    L, kind, case = native.load(), st["kind"], st["case"]
    if kind == "conv":
        rc = L.shkz_b200_conv3d_noalloc(case["nx"], case["ny"], case["nz"], case["c0"], case["c1"], case["cout"],
                                        case["planes"], _ptr(st["in0"]), _ptr(st["in1"]), _ptr(st["w"]),
                                        _ptr(st["b"]), 1, _ptr(st["out"]), None)
        if rc:
            raise native.ShkzError(rc, "conv3d_noalloc")
        return st["out"]
    if kind == "csr":
        st["ctx"].check(L.shkz_b200_solve_csr(st["ctx"].handle, len(st["b"]), st["indptr"].ctypes.data,
                                              st["indices"].ctypes.data, st["data"].ctypes.data, st["b"].ctypes.data,
                                              st["x"].ctypes.data, ctypes.byref(st["res"])), "solve_csr")
        return st["x"]
    if kind == "module":
        # project() keeps its own copies only where an array is not contiguous: give it this step's grids
        vel = MacGrid([v.copy() for v in st["vel"]], [m.copy() for m in st["act"]])
        st["solver"].project(case["dt"], vel, st["solid"], None, st["fluid"])
        p = st["solver"].get_pressure()
        return {"velocity": vel.values, "active": vel.active, "pressure": p.values, "unknowns": p.active}
    if kind == "network":
        z = st["solver"].learned_apply(st["r"])
        return {"z": z, "gradients": st["solver"].learned_backward(st["g"])}
    ctx, sc = st["ctx"], st["sc"]
    with torch.cuda.stream(st["stream"]):  # the calls update the velocity in place: this step's input
        for d in range(3):
            st["vel"][d].copy_(sc.vel[d], non_blocking=True)
            st["act"][d].copy_(sc.act[d], non_blocking=True)
    if kind == "splat":
        ctx.check(L.shkz_b200_splat_device(ctx.handle, ctypes.byref(st["args"])), "splat_device")
        return {"velocity": st["vel"], "active": st["act"]}
    if kind == "extend":
        ctx.check(L.shkz_b200_extend_velocity_device(ctx.handle, ctypes.byref(st["args"])), "extend_velocity_device")
        return {"velocity": st["vel"], "active": st["act"]}
    ctx.check(L.shkz_b200_project_device(ctx.handle, ctypes.byref(st["args"]), ctypes.byref(st["res"])),
              "project_device")
    return {"velocity": st["vel"], "active": st["act"], "pressure": st["pressure"], "unknowns": st["pressure_active"]}


def work(case):
    """Inputs read once and outputs written once. The iterations of a solve
    depend on the scene, so a solve counts its grids (its matrix) alone."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells, nodes = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    faces = (nx + 1) * ny * nz + nx * (ny + 1) * nz + nx * ny * (nz + 1)
    kind = case["kind"]
    solid = case.get("scene") in ("dambreak", "tank", "mixed")
    if kind == "conv":
        voxels, cin = cells, case["c0"] + case["c1"]
        return {"bytes": voxels * 2 * (case["c0"] + case["c1"] / 8 + case["cout"]) + 108 * cin * case["cout"],
                "flops": 2 * 27 * voxels * cin * case["cout"]}
    if kind == "csr":
        return {"bytes": cells * (8 + 7 * 16 + 16), "flops": 0}
    if kind == "network":
        # forward, input gradients and weight gradients of the liquid part
        share = 0.35
        macs = 27 * cells * (16 * 16 * 2 + 48 * 16 + 16 * 16 + 16
                             + (16 * 32 + 32 * 32 + 96 * 32 + 32 * 32) / 8 + (32 * 64 + 64 * 64) / 64)
        return {"bytes": cells * 12, "flops": 3 * 2 * macs * share}
    if kind == "splat":
        # the shell of the band around a surface of about one grid section
        count = case["per_cell"] * case["band"] * nx * nz
        return {"bytes": count * (65 if case["apic"] else 29) + 10 * 3 * (case["band"] + 1) * nx * nz, "flops": 0}
    if kind == "extend":
        return {"bytes": 10 * faces + (5 * nodes if solid else 0), "flops": 0}
    total = 10 * faces + 5 * cells + 5 * cells + (5 * nodes if solid else 0)
    return {"bytes": total + (4 * faces if case.get("moving") else 0), "flops": 0}


# ----------------------------------------------------------------------
# the same in 64 bits, with plain torch

def _polygon(v):
    """Area of the negative region of unit squares, v (m, 4) corner values in
    (0,0),(1,0),(1,1),(0,1) order: shoelace over kept corners and crossings."""
    qx, qy = (0.0, 1.0, 1.0, 0.0), (0.0, 0.0, 1.0, 1.0)
    pts = []
    for a in range(4):
        b = (a + 1) % 4
        zero = torch.zeros_like(v[:, a])
        pts.append((zero + qx[a], zero + qy[a], v[:, a] < 0))
        cross = v[:, a] * v[:, b] < 0
        t = torch.where(cross, v[:, a] / torch.where(cross, v[:, a] - v[:, b], zero + 1), zero)
        pts.append(((1 - t) * qx[a] + t * qx[b], (1 - t) * qy[a] + t * qy[b], cross))
    area = torch.zeros_like(v[:, 0])
    px, py, have = area.clone(), area.clone(), torch.zeros_like(pts[0][2])
    for turn in range(2):  # the second time round every point has a predecessor
        for x, y, on in pts:
            if turn:
                area = torch.where(on & have, area + px * y - py * x, area)
            px, py, have = torch.where(on, x, px), torch.where(on, y, py), have | on
    return 0.5 * area


def _face_geometry(sc, d, eps):
    """Open area and liquid fraction of the faces of axis d, as stored."""
    n = sc.n
    shape = [m + (a == d) for a, m in enumerate(n)][::-1]
    ax = 2 - d
    wall = torch.zeros(shape[ax], dtype=torch.bool, device=DEV)
    wall[0] = wall[-1] = True
    wall = wall.view([-1 if a == ax else 1 for a in range(3)]).expand(shape)
    exists = sc.solid is not None and bool(((sc.solid < 0) & (sc.solid_active != 0)).any())
    if not exists:
        area = torch.where(wall, 0.0, 1.0).double()
    else:
        lo, hi, al = slice(None, -1), slice(1, None), slice(None)
        corners = {0: [(lo, lo, al), (lo, hi, al), (hi, hi, al), (hi, lo, al)],
                   1: [(lo, al, lo), (lo, al, hi), (hi, al, hi), (hi, al, lo)],
                   2: [(al, lo, lo), (al, lo, hi), (al, hi, hi), (al, hi, lo)]}[d]
        act = torch.zeros(shape, dtype=torch.bool, device=DEV)
        neg = torch.zeros(shape, dtype=torch.int8, device=DEV)
        for c in corners:
            act |= sc.solid_active[c] != 0
            neg += (sc.solid[c] < 0).to(torch.int8)
        area = torch.where(neg == 4, 0.0, 1.0).double()
        mixed = (neg > 0) & (neg < 4)
        area[mixed] = 1.0 - _polygon(torch.stack([sc.solid[c][mixed].double() for c in corners], 1))
        area = torch.where(act & wall, torch.zeros_like(area), area)
        area = torch.where(act & (area != 0) & (area < eps), torch.full_like(area, eps), area)
    one = lambda t, i: t.narrow(ax, i, 1)  # noqa: E731
    f = sc.fluid.double()
    p1, p0 = torch.cat([f, one(f, n[d] - 1)], ax), torch.cat([one(f, 0), f], ax)
    cut = -torch.minimum(p0, p1) / (p1 - p0).abs().clamp(min=1e-300)
    rho = torch.where(p0 * p1 >= 0, ((p0 < 0) | (p1 < 0)).double(), cut)
    rho = torch.where((rho != 0) & (rho < eps), torch.full_like(rho, eps), rho)
    return area.float().double(), rho.float().double(), wall


def _exact_project(case, sc):
    n, dx, dt, eps = sc.n, sc.dx, case["dt"], 1e-2
    liquid = sc.fluid < 0
    geo = [_face_geometry(sc, d, eps) for d in range(3)]
    vel = [v.double() for v in sc.vel]
    if case.get("kappa"):
        f = sc.fluid.double()[None, None]
        g = torch.nn.functional.pad(f, (1,) * 6, mode="replicate")[0, 0]
        curv = (g[1:-1, 1:-1, 2:] + g[1:-1, 1:-1, :-2] + g[1:-1, 2:, 1:-1] + g[1:-1, :-2, 1:-1]
                + g[2:, 1:-1, 1:-1] + g[:-2, 1:-1, 1:-1] - 6 * f[0, 0]) / (dx * dx)
        for d in range(3):
            ax, (_, rho, _) = 2 - d, geo[d]
            up = lambda t: torch.cat([t, t.narrow(ax, n[d] - 1, 1)], ax)  # noqa: E731
            dn = lambda t: torch.cat([t.narrow(ax, 0, 1), t], ax)  # noqa: E731
            sgn = torch.where(up(sc.fluid) < 0, -1.0, 1.0).double()
            theta = torch.where(sgn < 0, 1 - rho, rho)
            face = theta * up(curv) + (1 - theta) * dn(curv)
            on = (sc.act[d] != 0) & (rho != 0) & (rho < 1)
            vel[d] = torch.where(on, vel[d] - sgn * dt / (dx * rho.clamp(min=eps)) * case["kappa"] * face, vel[d])
    weight, unknown = [], torch.zeros_like(liquid)
    diag = torch.zeros(liquid.shape, dtype=torch.float64, device=DEV)
    rhs = torch.zeros_like(diag)
    for d in range(3):
        ax, (area, rho, _) = 2 - d, geo[d]
        w = dt * area / (dx * dx * torch.where(rho != 0, rho, torch.ones_like(rho)))
        w = torch.where((area != 0) & (rho != 0), w, torch.zeros_like(w)).narrow(ax, 1, n[d] - 1)
        both = liquid.narrow(ax, 0, n[d] - 1) & liquid.narrow(ax, 1, n[d] - 1) & (w != 0)
        unknown.narrow(ax, 0, n[d] - 1).logical_or_(both)
        unknown.narrow(ax, 1, n[d] - 1).logical_or_(both)
        diag.narrow(ax, 0, n[d] - 1).add_(w)
        diag.narrow(ax, 1, n[d] - 1).add_(w)
        weight.append(torch.where(both, w, torch.zeros_like(w)))
        flux = area * vel[d] / dx
        if sc.svel is not None:
            flux = flux + (1 - area) * sc.svel[d].double() / dx
        rhs += flux.narrow(ax, 0, n[d]) - flux.narrow(ax, 1, n[d])
    rhs = torch.where(unknown, rhs, torch.zeros_like(rhs))
    diag = torch.where(unknown, diag, torch.ones_like(diag))

    def apply(p):
        q = diag * p
        for d in range(3):
            a, m = 2 - d, n[d] - 1
            q.narrow(a, 1, m).addcmul_(weight[d], p.narrow(a, 0, m), value=-1)
            q.narrow(a, 0, m).addcmul_(weight[d], p.narrow(a, 1, m), value=-1)
        return q

    # conjugate gradients, diagonal scaling; far below the tolerance of the case
    x, r = torch.zeros_like(rhs), rhs.clone()
    z = r / diag
    p, rz = z.clone(), (r * z).sum()
    stop = 1e-11 * float(rhs.abs().max())
    for it in range(6000):
        q = apply(p)
        alpha = rz / (p * q).sum()
        x.addcmul_(p, alpha)
        r.addcmul_(q, -alpha)
        if it % 20 == 0 and float(r.abs().max()) <= stop:
            break
        torch.div(r, diag, out=z)
        new = (r * z).sum()
        p.mul_(new / rz).add_(z)
        rz = new
    x = torch.where(unknown, x, torch.zeros_like(x))
    out, act = [], []
    for d in range(3):
        ax, (area, rho, wall) = 2 - d, geo[d]
        on = (sc.act[d] != 0) & (area != 0) & (rho != 0)
        grad = torch.zeros_like(vel[d])
        grad.narrow(ax, 1, n[d] - 1).copy_(x.narrow(ax, 1, n[d] - 1) - x.narrow(ax, 0, n[d] - 1))
        u = vel[d] - dt * grad / (torch.where(rho != 0, rho, torch.ones_like(rho)) * dx)
        u = torch.where(wall, sc.svel[d].double() if sc.svel is not None else torch.zeros_like(u), u)
        held = sc.act[d] != 0
        out.append(torch.where(on, u, torch.where(held, torch.zeros_like(u), vel[d])))
        act.append(on.to(torch.uint8))
    return {"velocity": out, "active": act, "pressure": x, "unknowns": unknown.to(torch.uint8)}


def _exact_splat(case, sc, rec):
    n, dx = sc.n, sc.dx
    rec = rec[rec[:, 17].view(torch.int32) == 0].double()
    p, mass = rec[:, 0:3], rec[:, 15]
    out = []
    for d in range(3):
        shape = [m + (a == d) for a, m in enumerate(n)]
        lo = [(p[:, a] / dx - (0.5 if a != d else 0.0)).floor().long() for a in range(3)]
        m = torch.zeros(shape[0] * shape[1] * shape[2], dtype=torch.float64, device=DEV)
        mom = torch.zeros_like(m)
        for o in range(8):
            i = [lo[a] + ((o >> a) & 1) for a in range(3)]
            # only faces of the cells' index range are activated
            ok = torch.stack([(i[a] >= 0) & (i[a] < n[a]) for a in range(3)]).all(0)
            pos = [(i[a].double() + (0.5 if a != d else 0.0)) * dx for a in range(3)]
            w = mass.clone()
            for a in range(3):
                w = w * (1 - (p[:, a] - pos[a]).abs() / dx).clamp(min=0)
            u = rec[:, 12 + d].clone()
            if case["apic"]:
                for a in range(3):
                    u = u + rec[:, 3 + 3 * d + a] * (pos[a] - p[:, a])
            at = (i[0] + shape[0] * (i[1] + shape[1] * i[2]))[ok]
            # every particle counts twice: the neighbour query visits each bucket twice
            m.index_add_(0, at, 2 * w[ok])
            mom.index_add_(0, at, 2 * (w * u)[ok])
        m, mom = m.view(shape[::-1]), mom.view(shape[::-1])
        g = torch.where(sc.act[d] != 0, (1 - m).clamp(min=0), torch.zeros_like(m))
        u = (g * sc.vel[d].double() + mom) / torch.where(m > 0, g + m, torch.ones_like(m))
        out.append(torch.where(m > 0, u, sc.vel[d].double()))
    return {"velocity": out, "active": [None] * 3}


def _sample(grid, pts):
    """Trilinear corner values (8, m) and their weight factors at index-space points."""
    D, H, W = grid.shape
    idx, frac = [], []
    for a, m in enumerate((W, H, D)):
        x = pts[a].clamp(0.0, m - 1.0)
        i = x.clamp(max=m - 2.0).floor()
        idx.append(i.long())
        frac.append(x - i)
    v = torch.stack([grid[idx[2] + (c >> 2), idx[1] + ((c >> 1) & 1), idx[0] + (c & 1)] for c in range(8)])
    return v, frac


def _weights(frac, along=None):
    got = []
    for c in range(8):
        w = torch.ones_like(frac[0])
        for a in range(3):
            b = (c >> a) & 1
            w = w * ((1.0 if b else -1.0) if a == along else (frac[a] if b else 1 - frac[a]))
        got.append(w)
    return torch.stack(got)


def _exact_extend(case, sc):
    vel, act = [v.double() for v in sc.vel], [m != 0 for m in sc.act]
    for d in range(3):
        for _ in range(case["width"]):
            s, k = torch.zeros_like(vel[d]), torch.zeros_like(vel[d])
            held = torch.where(act[d], vel[d], torch.zeros_like(vel[d]))
            for ax in range(3):
                m = held.shape[ax] - 1
                for a, b in ((0, 1), (1, 0)):
                    s.narrow(ax, a, m).add_(held.narrow(ax, b, m))
                    k.narrow(ax, a, m).add_(act[d].narrow(ax, b, m).double())
            new = ~act[d] & (k > 0)
            vel[d] = torch.where(new, s / k.clamp(min=1), vel[d])
            act[d] = act[d] | new
    held = [torch.where(a, v, torch.zeros_like(v)) for v, a in zip(vel, act)]
    out = []
    for d in range(3):
        u = vel[d].clone()
        if sc.solid is not None and bool(((sc.solid < 0) & (sc.solid_active != 0)).any()):
            at = act[d].nonzero()
            i = [at[:, 2 - a].double() + (0.0 if a == d else 0.5) for a in range(3)]
            sv, frac = _sample(sc.solid.double(), i)
            inside = (sv * _weights(frac)).sum(0) < 0
            at, i = at[inside], [c[inside] for c in i]
            sv, frac = sv[:, inside], [f[inside] for f in frac]
            nrm = torch.stack([(sv * _weights(frac, a)).sum(0) / sc.dx for a in range(3)])
            w = torch.stack([(lambda v, f: (v * _weights(f)).sum(0))(*_sample(
                held[c], [i[a] - (0.0 if a == c else 0.5) for a in range(3)])) for c in range(3)])
            un = (w * nrm).sum(0)
            hit = ((nrm ** 2).sum(0) != 0) & (un < 0)
            at = at[hit]
            u[at[:, 0], at[:, 1], at[:, 2]] = (w[d] - nrm[d] * un)[hit]
        if d == 1:
            lo, hi = u[:, 0, :], u[:, -1, :]
            lo.copy_(torch.where(act[d][:, 0, :] & (lo < 0), torch.zeros_like(lo), lo))
            hi.copy_(torch.where(act[d][:, -1, :] & (hi > 0), torch.zeros_like(hi), hi))
        out.append(u)
    return {"velocity": out, "active": [a.to(torch.uint8) for a in act]}


def _exact_csr(case, seed):
    indptr, indices, data, b = _csr(case, seed)
    n = len(b)
    A = torch.sparse_csr_tensor(torch.from_numpy(indptr), torch.from_numpy(indices), torch.from_numpy(data),
                                size=(n, n), dtype=torch.float64).to(DEV)
    b = torch.from_numpy(b).to(DEV)
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    rows = torch.from_numpy(np.repeat(np.arange(n), np.diff(indptr))).to(DEV)
    on = rows == torch.from_numpy(indices).to(DEV)
    diag[rows[on]] = torch.from_numpy(data).to(DEV)[on]
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz = z.clone(), r @ z
    for _ in range(4000):
        q = A @ p
        alpha = rz / (p @ q)
        x, r = x + alpha * p, r - alpha * q
        if float(r.abs().max()) <= 1e-13 * float(b.abs().max()):
            break
        z = r / diag
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x


def _exact_conv(case, seed):
    in0, in1, w, b = _conv_inputs(case, seed)
    x = in0.double()
    if in1 is not None:
        up = in1.double()
        for a in range(3):
            up = up.repeat_interleave(2, a)
        x = torch.cat([x, up], -1)
    nz, ny, nx, _ = x.shape
    x = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    out = torch.zeros((nz, ny, nx, case["cout"]), dtype=torch.float64, device=DEV)
    for t in range(27):
        dz, dy, dx_ = t // 9, (t // 3) % 3, t % 3
        out += x[dz:dz + nz, dy:dy + ny, dx_:dx_ + nx] @ w[t].double().T
    return (out + b.double()).clamp(min=0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "conv":
        return _exact_conv(case, seed)
    if kind == "csr":
        return _exact_csr(case, seed)
    if kind == "network" or case["nx"] * case["ny"] * case["nz"] > 400 ** 3:
        return None  # 16-bit activations throughout; the largest solve takes too long
    sc = Scene(case, seed)
    if kind == "splat":
        return _exact_splat(case, sc, _particles(sc, case, seed))
    if kind == "extend":
        return _exact_extend(case, sc)
    return _exact_project(case, sc)
