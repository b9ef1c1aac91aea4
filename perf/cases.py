"""The measured workloads: what a program that uses the solver has it do, through the public
entry points of the Python binding (incompflow-cuda_b200/python/ifc.py).

Most cases are a solve continued from a given state for a fixed number of outer iterations (the
bulk of every solve to convergence is such iterations on a developed flow): the program keeps
its start fields on the device, copies them into the handle's fields (Solver.device_ptr) on the
handle's stream, and reads the results there.  `exact` is the same method in 64 bits, written
with whole-array torch operations.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "incompflow-cuda_b200", "python"))
import ifc  # noqa: E402

E, W, N, S, T, B = range(6)


def listed():
    return [
        # a small closed cavity, odd sizes: two tiles' worth of cells, so launches and
        # barriers are most of the time (parameter studies, tests)
        dict(name="cavity2d_33x31", kind="flow", bc="cavity", dim=2, nx=33, ny=31, nz=1, prec="f", conv="upwind",
             iters=10),
        # a whole solve() call to convergence by the default rule, the 64^2 cavity at Re 100
        dict(name="solve_cavity2d_64", kind="solve", bc="cavity", dim=2, nx=64, ny=64, nz=1, prec="f", conv="upwind",
             iters=20000),
        # the headline workload: the 512x128 channel, one step of 100 outer iterations
        dict(name="channel2d_512x128", kind="flow", bc="channel", dim=2, nx=512, ny=128, nz=1, prec="f",
             conv="upwind", iters=100),
        # the grid of the shipped configuration (1024x256)
        dict(name="channel2d_1024x256", kind="flow", bc="channel", dim=2, nx=1024, ny=256, nz=1, prec="f",
             conv="upwind", iters=20),
        # a large 2D grid, as the slab record of the benchmark has it
        dict(name="channel2d_4096x2048", kind="flow", bc="channel", dim=2, nx=4096, ny=2048, nz=1, prec="f",
             conv="upwind", iters=4),
        # double precision with higher-order convection on a ragged grid (reference solutions)
        dict(name="channel2d_500x190_f64_quick", kind="flow", bc="channel", dim=2, nx=500, ny=190, nz=1, prec="d",
             conv="quick", iters=20),
        # the 128^3 lid-driven cube of the precision study
        dict(name="cavity3d_128", kind="flow", bc="cavity", dim=3, nx=128, ny=128, nz=128, prec="f", conv="upwind",
             iters=5),
        # its double-precision counterpart with higher-order convection, ragged
        dict(name="cavity3d_97x89x101_f64_quick", kind="flow", bc="cavity", dim=3, nx=97, ny=89, nz=101, prec="d",
             conv="quick", iters=4),
        # a large 3D grid: twice the README's 3D memory example in each direction but x
        dict(name="cavity3d_256", kind="flow", bc="cavity", dim=3, nx=256, ny=256, nz=256, prec="f", conv="upwind",
             iters=2),
        # the temperature on a finished channel flow, a fixed number of sweeps
        dict(name="energy2d_512x128", kind="energy", bc="channel", dim=2, nx=512, ny=128, nz=1, prec="f",
             conv="upwind", iters=400),
        # the gradient of a design loop: reverse passes of the discrete adjoint, 256x64 channel
        dict(name="adjoint_256x64", kind="adjoint", bc="channel", dim=2, nx=256, ny=64, nz=1, prec="f",
             conv="upwind", iters=150),
        # many uneven cavities at once, sizes and Reynolds numbers of the batched workload
        dict(name="batch_48", kind="batch", bc="cavity", dim=2, nx=256, ny=256, nz=1, prec="f", conv="upwind",
             count=48, iters=60),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow2", "flow2", "flow2", "flow3", "flow3", "energy", "adjoint", "batch"])
    prec = rng.choice(["f", "f", "f", "d"])
    bc = rng.choice(["channel", "cavity"])
    c = dict(kind="flow", bc=bc, dim=2, nz=1, prec=prec, conv=rng.choice(["upwind", "upwind", "quick", "van_leer"]))
    if kind == "flow2":
        c.update(nx=_log_int(rng, 24, 4096), ny=_log_int(rng, 16, 1024))
        # at most 4e6 cells x iterations in all (half of that in double precision)
        c["iters"] = max(1, min(60, int((4e6 if prec == "f" else 2e6) / (c["nx"] * c["ny"]))))
    elif kind == "flow3":
        c.update(dim=3, nx=_log_int(rng, 12, 160), ny=_log_int(rng, 12, 160), nz=_log_int(rng, 12, 160))
        c["iters"] = max(1, min(10, int((6e6 if prec == "f" else 3e6) / (c["nx"] * c["ny"] * c["nz"]))))
    elif kind == "energy":
        d3 = rng.random() < 0.4
        c.update(kind="energy", conv="upwind", dim=3 if d3 else 2)
        if d3:
            c.update(nx=_log_int(rng, 12, 128), ny=_log_int(rng, 12, 128), nz=_log_int(rng, 12, 128))
        else:
            c.update(nx=_log_int(rng, 24, 1024), ny=_log_int(rng, 16, 256))
        c["iters"] = rng.randrange(50, 401)
    elif kind == "adjoint":
        c.update(kind="adjoint", bc="channel", conv="upwind", nx=_log_int(rng, 32, 256), ny=_log_int(rng, 16, 80),
                 iters=rng.randrange(40, 121))
    else:
        c.update(kind="batch", bc="cavity", conv="upwind", nx=256, ny=256, count=rng.randrange(4, 33), prec=prec,
                 iters=rng.randrange(20, 51))
        if prec == "d":
            c["iters"] = max(10, c["iters"] // 2)
    return c


# ---------------------------------------------------------------- inputs

def _config(c):
    """The library's configuration of a case."""
    if c["bc"] == "channel":
        cfg = ifc.channel2d(c["nx"], c["ny"])
        if c["dim"] == 3:
            cfg.update(dim=3, nz=c["nz"], zmin=-0.0125, zmax=0.0125, nIter_w=10)
    elif c["dim"] == 3:
        cfg = ifc.cavity3d(c["nx"], nx=c["nx"], ny=c["ny"], nz=c["nz"])
    else:
        cfg = ifc.cavity2d(c["nx"], ny=c["ny"])
    cfg["precision"] = c["prec"]
    cfg["convection_scheme"] = c["conv"]
    if c["kind"] == "solve":
        cfg["numOuterIter"] = c["iters"]
    return cfg


def _batch_cases(c, seed):
    # the workload's sizes; the fluids from the seed, Re log-uniform in [10, 1000]
    cfgs = ifc.batch_cases(c["count"], seed=0)
    res = 10.0 ** np.random.default_rng(int(seed)).uniform(1.0, 3.0, c["count"])
    for k, re in zip(cfgs, res):
        k["dynamicViscosity"] = float(1.0 / re)
        k["numOuterIter"] = c["iters"]
        k["precision"] = c["prec"]
    return cfgs


def _dtype(c):
    return torch.float64 if c["prec"] == "d" else torch.float32


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _smooth(g, dim, x, y, z):
    """A smooth random function of order one: a few low modes with random phases."""
    out = torch.zeros_like(x + y + z)
    r = torch.rand(4, 7, generator=g, device=x.device, dtype=torch.float64).cpu().tolist()
    for q in r:
        kx, ky, kz = 1 + int(3 * q[0]), 1 + int(3 * q[1]), 1 + int(3 * q[2])
        m = torch.cos(math.pi * kx * x + 6.2832 * q[3]) * torch.cos(math.pi * ky * y + 6.2832 * q[4])
        if dim == 3:
            m = m * torch.cos(math.pi * kz * z + 6.2832 * q[5])
        out = out + (q[6] - 0.5) * m
    return out


def _fields(c, seed):
    """Start fields u, v, (w,) p: a developed-looking flow (parabolic channel flow, or the recirculation
    of a driven cavity) with smooth deviations and a little noise, all from the seed."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    cfg = _config(c)
    dim, nx, ny, nz = c["dim"], c["nx"], c["ny"], c["nz"]
    f64 = dict(dtype=torch.float64, device=dev)
    x = ((torch.arange(nx, **f64) + 0.5) / nx).view(1, 1, nx)
    y = ((torch.arange(ny, **f64) + 0.5) / ny).view(1, ny, 1)
    z = ((torch.arange(nz, **f64) + 0.5) / nz).view(nz, 1, 1)
    one = torch.ones(nz, ny, nx, **f64)

    def noise():
        return torch.randn(nz, ny, nx, generator=g, **f64)

    if c["bc"] == "channel":
        U = 0.001
        rho = cfg["density"]
        prof = 6.0 * y * (1.0 - y) * (6.0 * z * (1.0 - z) / 1.44 if dim == 3 else 1.0)
        wall = 4.0 * y * (1.0 - y)
        u = U * (prof * (1.0 + 0.05 * _smooth(g, dim, x, y, z)) * one + 0.002 * noise())
        v = U * (0.05 * wall * _smooth(g, dim, x, y, z) * one + 0.002 * noise())
        w = U * (0.05 * wall * _smooth(g, dim, x, y, z) * one + 0.002 * noise())
        p = rho * U * U * (4.0 * (1.0 - x) + 0.2 * _smooth(g, dim, x, y, z) + 0.002 * noise())
    else:
        a, b = x, (z if dim == 3 else y)   # the plane in which the lid drives the flow
        sa, sb = torch.sin(math.pi * a), torch.sin(math.pi * b)
        amp = 0.25 * (torch.sin(math.pi * y) if dim == 3 else 1.0)
        u = amp * (-2.0 * sa * sa * sb * torch.cos(math.pi * b)) * one
        up = amp * (2.0 * sa * torch.cos(math.pi * a) * sb * sb) * one
        u = u + 0.02 * sa * sb * _smooth(g, dim, x, y, z) + 0.0005 * noise()
        up = up + 0.02 * sa * sb * _smooth(g, dim, x, y, z) + 0.0005 * noise()
        side = 0.02 * sa * sb * _smooth(g, dim, x, y, z) + 0.0005 * noise()
        v, w = (side, up) if dim == 3 else (up, side)
        p = 0.05 * _smooth(g, dim, x, y, z) * one + 0.0005 * noise()
    out = {"u": u, "v": v, "p": p}
    if dim == 3:
        out["w"] = w
    return {k: t.to(_dtype(c)).contiguous() for k, t in out.items()}


def _profile(c, seed):
    """The inlet profile of a design iterate: the uniform inlet with smooth deviations."""
    y = (np.arange(c["ny"]) + 0.5) / c["ny"]
    r = np.random.default_rng(int(seed)).normal(0.0, 1.0, 4)
    return 0.001 * (1.0 + 0.05 * sum(r[k] * np.cos(math.pi * (k + 1) * y) for k in range(4)))


def _mass_fluxes(c, seed):
    """Face velocities of a divergence-free flow (2D stream function; in 3D the same in every plane) and a
    start temperature, for the energy equation."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    cfg = _config(c)
    dim, nx, ny, nz = c["dim"], c["nx"], c["ny"], c["nz"]
    f64 = dict(dtype=torch.float64, device=dev)
    xn = (torch.arange(nx + 1, **f64) / nx).view(1, 1, nx + 1)
    yn = (torch.arange(ny + 1, **f64) / ny).view(1, ny + 1, 1)
    dx, dy = (cfg["xmax"] - cfg["xmin"]) / nx, (cfg["ymax"] - cfg["ymin"]) / ny
    H = cfg["ymax"] - cfg["ymin"]
    bump = (torch.sin(math.pi * xn) * torch.sin(math.pi * yn)) ** 2
    dev_ = 0.1 * bump * _smooth(g, 2, xn, yn, torch.zeros(1, 1, 1, **f64))
    if c["bc"] == "channel":
        psi = 0.001 * H * (yn * yn * (3.0 - 2.0 * yn) + dev_)
    else:
        psi = 0.25 * H * (bump + dev_)
    uf = ((psi[:, 1:, :] - psi[:, :-1, :]) / dy).expand(nz, ny, nx + 1)
    vf = (-(psi[:, :, 1:] - psi[:, :, :-1]) / dx).expand(nz, ny + 1, nx)
    temp = 320.0 + 20.0 * torch.randn(nz, ny, nx, generator=g, **f64)
    out = {"uf": uf, "vf": vf, "T": temp}
    if dim == 3:
        out["wf"] = torch.zeros(nz + 1, ny, nx, **f64)
    return {k: t.to(_dtype(c)).contiguous() for k, t in out.items()}


# ---------------------------------------------------------------- one pass

class _OnDevice:
    """A field of a handle as CUDA array interface; keeps the handle alive while a view of it lives."""

    def __init__(self, solver, name):
        self.solver = solver
        dt = np.dtype(solver.dtype)
        n = solver.field_size(name) // dt.itemsize
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": dt.str, "version": 3,
                                         "data": (solver.device_ptr(name), False)}


def _view(solver, name):
    return torch.as_tensor(_OnDevice(solver, name), device="cuda")


class _State:
    pass


def prepare(case, seed):
    c = case
    s = _State()
    s.case = c
    if c["kind"] == "batch":
        s.cfgs = _batch_cases(c, seed)
        return s
    s.stream = torch.cuda.Stream()
    cfg = dict(_config(c), stream=s.stream.cuda_stream)
    if c["kind"] == "adjoint":
        cfg["inlet_profile"] = _profile(c, seed)
    start = _mass_fluxes(c, seed) if c["kind"] == "energy" else _fields(c, seed)
    s.start = {k: t.reshape(-1) for k, t in start.items()}
    torch.cuda.synchronize()
    s.solver = ifc.Solver(cfg)
    names = list(s.start)
    if c["kind"] in ("flow", "solve"):
        names += ["uf", "vf"] + (["wf"] if c["dim"] == 3 else [])
    s.views = {k: _view(s.solver, k) for k in names}
    if c["kind"] == "adjoint":       # the flow whose gradient is asked for
        _restart(s)
        s.solver.iterate(200)
    elif c["kind"] == "energy":
        for k in s.start:
            s.views[k].copy_(s.start[k])
        torch.cuda.synchronize()
    return s


def _restart(s):
    """A new solve from the start fields: counters and faces reset, fields copied on the handle's stream."""
    s.solver.set_uniform()
    with torch.cuda.stream(s.stream):
        for k, t in s.start.items():
            s.views[k].copy_(t)


def run(state):
    s, c = state, state.case
    if c["kind"] == "batch":
        results, fields, _ = ifc.batch_solve(s.cfgs)
        return {"fields": [np.concatenate([f["u"], f["v"], f["p"]]) for f in fields],
                "outer_iterations": np.array([r["outer_iterations"] for r in results])}
    if c["kind"] == "adjoint":
        dtheta, r = s.solver.adjoint(max_iter=c["iters"], tol=0.0)
        return {"dJ_dtheta": dtheta, "dJ_dmu": np.array([r["dJ_dmu"]]), "objective": np.array([r["objective"]])}
    if c["kind"] == "energy":
        with torch.cuda.stream(s.stream):
            s.views["T"].copy_(s.start["T"])
        r = s.solver.solve_energy(max_sweeps=c["iters"], tol=0.0)
        return {"T": s.views["T"], "sweeps": int(r["sweeps"])}
    _restart(s)
    st = s.solver.solve() if c["kind"] == "solve" else s.solver.iterate(c["iters"])
    return {"fields": dict(s.views), "outer_iterations": int(st["outer_iterations"])}


# ---------------------------------------------------------------- work

def work(case):
    """Bytes: start fields in, results out.  Operations: every relaxed point update of the method (four or six
    products and differences, one division, the relaxation), and the assembly, Rhie-Chow, link and correction
    arithmetic of each cell and outer iteration."""
    c = case
    it, item = c["iters"], 8 if c["prec"] == "d" else 4
    cells = c["nx"] * c["ny"] * c["nz"]
    upd = 12.0 if c["dim"] == 2 else 16.0
    if c["kind"] == "batch":
        total = sum(k["nx"] * k["ny"] for k in _batch_cases(c, 0))
        return {"bytes": 3.0 * item * total, "flops": total * it * (upd * 60 + 120.0)}
    if c["kind"] == "energy":
        faces = 3 if c["dim"] == 3 else 2
        return {"bytes": item * cells * (2.0 + faces), "flops": cells * it * upd}
    if c["kind"] == "adjoint":
        # primal state in, gradient out; transposed sweeps of u, v (10 each) and p' (20), 9 operations each
        return {"bytes": item * cells * 5.0 + 8.0 * c["ny"], "flops": cells * it * (9.0 * 40 + 200.0)}
    if c["kind"] == "solve":
        it = 800  # about what this flow takes to converge
    cfg = _config(c)
    sweeps = cfg["nIter_u"] + cfg["nIter_v"] + cfg["nIter_p"] + (cfg["nIter_w"] if c["dim"] == 3 else 0)
    return {"bytes": item * cells * (1.0 + c["dim"]) * 2 + item * cells * c["dim"],
            "flops": cells * it * (upd * sweeps + (120.0 if c["dim"] == 2 else 190.0))}


# ---------------------------------------------------------------- the method in 64 bits

def _sh(a, axis, d, fill=0.0):
    """a shifted so that out[i] = a[i + d] along the axis, `fill` outside."""
    out = torch.full_like(a, fill)
    n = a.shape[axis]
    if abs(d) >= n:
        return out
    if d > 0:
        out.narrow(axis, 0, n - d).copy_(a.narrow(axis, d, n - d))
    else:
        out.narrow(axis, -d, n + d).copy_(a.narrow(axis, 0, n + d))
    return out


class _Exact:
    """The SIMPLE iteration (red-black sweeps, Rhie-Chow, relaxed corrections) on (nz, ny, nx) arrays."""

    AX = {"x": 2, "y": 1, "z": 0}

    def __init__(self, c):
        cfg = self.cfg = _config(c)
        self.c, self.dim = c, c["dim"]
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        dx, dy = (cfg["xmax"] - cfg["xmin"]) / nx, (cfg["ymax"] - cfg["ymin"]) / ny
        dz = (cfg["zmax"] - cfg["zmin"]) / nz
        self.A = {"x": dy * dz, "y": dz * dx, "z": dx * dy}
        self.d = {"x": dx, "y": dy, "z": dz}
        self.rho, self.mu = cfg["density"], cfg["dynamicViscosity"]
        self.axes = ["x", "y", "z"][: self.dim]
        self.bc, self.val = cfg["velBC_type"], cfg["velBC_val"]
        dev = _device()
        i, j, k = (torch.arange(n, device=dev) for n in (nx, ny, nz))
        self.red = ((i.view(1, 1, -1) + j.view(1, -1, 1) + k.view(-1, 1, 1)) % 2) == 0
        self.faces = {"x": (W, E), "y": (S, N), "z": (B, T)}  # low, high face of each axis
        self.comp = {"x": 0, "y": 1, "z": 2}

    def low(self, F, ax):   # the low face of each cell
        return F.narrow(self.AX[ax], 0, F.shape[self.AX[ax]] - 1)

    def high(self, F, ax):
        return F.narrow(self.AX[ax], 1, F.shape[self.AX[ax]] - 1)

    def face_bcs(self, F, ax, phi):
        a = self.AX[ax]
        n = F.shape[a] - 1
        for end, face in ((0, self.faces[ax][0]), (n, self.faces[ax][1])):
            t = self.bc[face]
            sl = F.narrow(a, end, 1)
            if t == ifc.WALL:
                sl.zero_()
            elif t == ifc.INLET:
                sl.fill_(self.val[face][self.comp[ax]])
            else:
                sl.copy_(phi.narrow(a, 0 if end == 0 else n - 1, 1))

    def links(self, F, D):
        """Upwind and diffusion links of every cell: {(axis, +1/-1): array}, and the diagonal."""
        a, aC = {}, 0.0
        for ax in self.axes:
            a[ax, 1] = self.rho * self.A[ax] * torch.clamp(self.high(F[ax], ax), max=0.0) - D[ax]
            a[ax, -1] = self.rho * self.A[ax] * torch.clamp(-self.low(F[ax], ax), max=0.0) - D[ax]
            aC = aC - (a[ax, 1] + a[ax, -1])
        return a, aC

    def fold(self, a, aC, b, kinds, values):
        """Boundary faces into diagonal and sources, in the order E W N S T B."""
        for face in (E, W, N, S, T, B)[: 2 * self.dim]:
            ax = {E: "x", W: "x", N: "y", S: "y", T: "z", B: "z"}[face]
            d = 1 if face in (E, N, T) else -1
            x = self.AX[ax]
            at = a[ax, d].shape[x] - 1 if d > 0 else 0
            e = a[ax, d].narrow(x, at, 1).clone()
            c = aC.narrow(x, at, 1)
            if kinds[face] == "open":
                c += e
            else:
                c -= 2 * e
                a[ax, -d].narrow(x, at, 1).add_(e / 3)
                for m, src in enumerate(b):
                    src.narrow(x, at, 1).sub_(8.0 / 3.0 * e * values[face][m])
            a[ax, d].narrow(x, at, 1).zero_()

    def sweep(self, phi, a, aC, b, relax):
        for color in (self.red, ~self.red):
            s = b
            for (ax, d), l in a.items():
                s = s - l * _sh(phi, self.AX[ax], d)
            phi = torch.where(color, phi + relax * (s / aC - phi), phi)
        return phi

    def side(self, p, ax, d):
        """p of the neighbour; at the domain's edge the cell's own (closed face) or 0 (open)."""
        x = self.AX[ax]
        out = _sh(p, x, d)
        face = self.faces[ax][1 if d > 0 else 0]
        if self.bc[face] != ifc.OUTLET:
            at = p.shape[x] - 1 if d > 0 else 0
            out.narrow(x, at, 1).copy_(p.narrow(x, at, 1))
        return out

    def deferred(self, phi, F):
        """Higher-order minus upwind convection of phi, per cell."""
        total = torch.zeros_like(phi)
        for ax in self.axes:
            x, n = self.AX[ax], phi.shape[self.AX[ax]]
            fl = self.rho * F[ax].narrow(x, 1, n - 1) * self.A[ax]       # interior faces
            L, R = phi.narrow(x, 0, n - 1), phi.narrow(x, 1, n - 1)
            LL, RR = _sh(L, x, -1), _sh(R, x, 1)
            pos = fl > 0
            du = torch.where(pos, L - LL, R - RR)
            dd = torch.where(pos, R - L, L - R)
            if self.c["conv"] == "quick":
                lim = (3 * dd + du) / 4
            else:   # van Leer
                ok = du * dd > 0
                lim = torch.where(ok, 2 * du * dd / torch.where(ok, du + dd, torch.ones_like(du)), torch.zeros_like(du))
            q = fl * 0.5 * lim
            idx = torch.arange(n - 1, device=phi.device).view([-1 if k == x else 1 for k in range(3)])
            q = torch.where((pos & (idx == 0)) | (~pos & (idx == n - 2)) | (fl == 0), torch.zeros_like(q), q)
            total.narrow(x, 1, n - 1).add_(q)
            total.narrow(x, 0, n - 1).sub_(q)
        return total

    def flow(self, start, iters):
        cfg, dim = self.cfg, self.dim
        vel = [start[k].clone() for k in ("u", "v", "w")[:dim]]
        p = start["p"].clone()
        relax = [cfg["relax_u"], cfg["relax_v"], cfg["relax_w"]]
        sweeps = [cfg["nIter_u"], cfg["nIter_v"], cfg["nIter_w"]]
        D = {ax: self.mu * self.A[ax] / self.d[ax] for ax in self.axes}
        kinds = {f: "open" if self.bc[f] == ifc.OUTLET else "wall" for f in range(6)}
        F = {}
        for m, ax in enumerate(self.axes):
            x = self.AX[ax]
            shape = list(p.shape)
            shape[x] += 1
            F[ax] = torch.zeros(shape, dtype=p.dtype, device=p.device)
            n = p.shape[x]
            F[ax].narrow(x, 1, n - 1).copy_((vel[m].narrow(x, 0, n - 1) + vel[m].narrow(x, 1, n - 1)) / 2)
            self.face_bcs(F[ax], ax, vel[m])
        pin = all(self.bc[f] != ifc.OUTLET for f in range(2 * dim))
        for _ in range(iters):
            dc = [self.deferred(vel[m], F) for m in range(dim)] if self.c["conv"] != "upwind" else None
            a, aC = self.links(F, D)
            b = [0.5 * (self.side(p, ax, -1) - self.side(p, ax, 1)) * self.A[ax] for ax in self.axes]
            self.fold(a, aC, b, kinds, self.val)
            for m in range(dim):
                src = b[m] + dc[m] if dc else b[m]
                for _s in range(sweeps[m]):
                    vel[m] = self.sweep(vel[m], a, aC, src, relax[m])
            r = 1.0 / aC
            mass = torch.zeros_like(p)
            pa, pC = {}, 0.0
            for m, ax in enumerate(self.axes):
                x, A, n = self.AX[ax], self.A[ax], p.shape[self.AX[ax]]
                lo, hi = (lambda t: t.narrow(x, 0, n - 1)), (lambda t: t.narrow(x, 1, n - 1))
                grad = (self.side(p, ax, 1) - self.side(p, ax, -1)) * A * r / 4    # (p_E - p_W) A / (4 aC)
                sr = lo(r) + hi(r)
                F[ax].narrow(x, 1, n - 1).copy_(0.5 * (lo(vel[m]) + hi(vel[m])) + lo(grad) + hi(grad)
                                                + 0.5 * sr * (lo(p) - hi(p)) * A)
                self.face_bcs(F[ax], ax, vel[m])
                mass += self.rho * A * (self.low(F[ax], ax) - self.high(F[ax], ax))
                link = -0.5 * self.rho * A * A * sr
                pa[ax, 1], pa[ax, -1] = torch.zeros_like(p), torch.zeros_like(p)
                lo(pa[ax, 1]).copy_(link)
                hi(pa[ax, -1]).copy_(link)
                pC = pC - (pa[ax, 1] + pa[ax, -1])
            pc = torch.zeros_like(p)
            for _s in range(cfg["nIter_p"]):
                pc = self.sweep(pc, pa, pC, mass, cfg["relax_p"])
            if pin:
                pc = pc - pc.mean()
            p = p + cfg["relax_p"] * pc
            for m, ax in enumerate(self.axes):
                x, A, n = self.AX[ax], self.A[ax], p.shape[self.AX[ax]]
                lo, hi = (lambda t: t.narrow(x, 0, n - 1)), (lambda t: t.narrow(x, 1, n - 1))
                vel[m] = vel[m] + 0.5 * relax[m] * (self.side(pc, ax, -1) - self.side(pc, ax, 1)) * A * r
                F[ax].narrow(x, 1, n - 1).add_(0.5 * relax[m] * (lo(r) + hi(r)) * (lo(pc) - hi(pc)) * A)
                self.face_bcs(F[ax], ax, vel[m])
        out = dict(zip(("u", "v", "w"), vel), p=p)
        out.update({ax_name: F[ax] for ax, ax_name in zip(self.axes, ("uf", "vf", "wf"))})
        return out

    def energy(self, given, sweeps):
        F = {ax: given[k] for ax, k in zip(self.axes, ("uf", "vf", "wf"))}
        gam = self.cfg["thermalConductivity"] / self.cfg["specificHeatCapacity"]
        a, aC = self.links(F, {ax: gam * self.A[ax] / self.d[ax] for ax in self.axes})
        b = [torch.zeros_like(given["T"])]
        kinds = {f: "open" if self.cfg["TempBC_type"][f] else "wall" for f in range(6)}
        self.fold(a, aC, b, kinds, [[v] for v in self.cfg["TempBC_val"]])
        t = given["T"].clone()
        for _ in range(sweeps):
            t = self.sweep(t, a, aC, b[0], 1.0)
        return t


def exact(case, seed):
    c = case
    if c["kind"] == "energy":
        given = {k: t.double() for k, t in _mass_fluxes(c, seed).items()}
        return {"T": _Exact(c).energy(given, c["iters"]).reshape(-1), "sweeps": None}
    if c["kind"] == "flow":
        start = {k: t.double() for k, t in _fields(c, seed).items()}
        out = _Exact(c).flow(start, c["iters"])
        return {"fields": {k: t.reshape(-1) for k, t in out.items()}, "outer_iterations": None}
    return None     # whole solves, batches and gradients: over 20 seconds this way
