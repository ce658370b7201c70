"""The workloads this library is used for, each as one call a program makes.

A case is a dict of plain values.  kind says which public entry points it goes
through:

  poisson    ibpm_lap_inv_noalloc on a caller's device buffers
  static     GpuCnabSolver on static bodies: `steps` advance_ calls, the forces
             read after each, then the vorticity of every level (what a saver
             that writes every `steps` steps does)
  moving     the same with a pitching and plunging plate (CG force solve)
  ensemble   an Ensemble of `count` cases advanced `steps` steps in one call,
             then the forces and the level-1 vorticity of every case
  solve      ib.solve on a new geometry: the solver's construction (B and its
             inverse) and `steps` steps, as a sweep over shapes does

FP32 and mixed engines are used for their fields (their forces carry noise of
1e-3 that the force system amplifies from FP32 rounding), so those cases return
the vorticity, in FP32, after a few steps; FP64 cases return forces too.

`exact` restates the method in plain torch (float64, dense sine matrices for
the transforms), sharing no code with the package.
"""
import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import load_package

ib = load_package()

# transform lengths the library takes (even, 2^a 3^b 5^c, at most 1024) that
# users pick: powers of two and round numbers
SIZES = [64, 72, 80, 96, 100, 108, 120, 128, 144, 150, 160, 180, 192, 200, 216, 240, 256, 270, 288, 300, 320, 324, 360,
         384, 400, 432, 450, 480, 500, 512, 540, 576, 600, 640, 648, 720, 750, 768, 800, 810, 864, 900, 960, 1000, 1024]


def _static(name, nx, ny, levels, h, body, Re, dt, steps, precision="fp64", grid="fixed"):
    return dict(name=name, kind="static", nx=nx, ny=ny, levels=levels, h=h, body=body, Re=Re, dt=dt, steps=steps,
                precision=precision, grid=grid)


def listed():
    return [
        # one Poisson solve inside another program's loop (smallest call)
        dict(name="poisson_384x256", kind="poisson", nx=384, ny=256),
        # a first look at a flow on a small grid: latency only
        _static("cylinder_64", 64, 64, 3, 4 / 64, "cylinder", 100.0, 0.0125, 10),
        # the 200 x 200 cylinder that also runs on a CPU
        _static("cylinder_200", 200, 200, 3, 0.02, "cylinder", 100.0, 0.004, 10),
        # ragged sizes (factors 3 and 5), two bodies
        _static("two_bodies_360x300", 360, 300, 4, 0.0125, "both", 150.0, 0.0025, 10),
        # a body-fixed, moving grid
        _static("moving_grid_256", 256, 256, 3, 4 / 256, "plate", 100.0, 0.003, 10, grid="moving"),
        # the headline workload: 1024 x 1024 x 5 levels, 628 points, noise, a saver every 40 steps
        _static("cylinder_1024", 1024, 1024, 5, 0.005, "cylinder", 100.0, 0.001, 40),
        # the flat plate at 30 degrees in the FP32 engine, for its fields
        _static("plate_1024_fp32", 1024, 1024, 5, 0.005, "plate", 200.0, 0.001, 6, precision="fp32"),
        # parameter studies: batched groups of cases
        dict(name="ensemble_16_fp64", kind="ensemble", count=16, precision="fp64", steps=10),
        dict(name="ensemble_48_fp32", kind="ensemble", count=48, precision="fp32", steps=8),
        # the moving plate, plain CG at the default tolerance
        dict(name="pitching_512_cg", kind="moving", n=512, levels=4, h=0.01, k=0.55, Re=500.0, dt=0.002, steps=2,
             start="previous", depth=8, products=0),
        # the moving plate, preconditioned CG with the tensor-core rebuild every 8 steps
        dict(name="pitching_512_precond", kind="moving", n=512, levels=4, h=0.01, k=0.55, Re=500.0, dt=0.002, steps=16,
             start="preconditioned_extrapolated", depth=8, products=3),
        # a sweep over geometries: construction and the first steps of a new one
        dict(name="solve_256", kind="solve", nx=256, ny=256, levels=3, h=0.015625, body="plate", Re=100.0, dt=0.003,
             steps=5),
    ]


def _log_size(rng, lo, hi):
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((s for s in SIZES if lo <= s <= hi), key=lambda s: abs(math.log(s / want)))


def draw(rng):
    kind = rng.choice(["poisson", "static", "static", "static", "static", "ensemble", "moving", "moving", "solve"])
    if kind == "poisson":
        while True:
            nx, ny = _log_size(rng, 64, 1024), _log_size(rng, 64, 1024)
            if (nx - 1) * (ny - 1) <= 262144:
                return dict(kind=kind, nx=nx, ny=ny)
    if kind in ("static", "solve"):
        nx = _log_size(rng, 64, 1024 if kind == "static" else 400)
        ny = _log_size(rng, max(64, nx // 2), min(nx * 2, 1024 if kind == "static" else 400))
        levels = rng.randint(1, 5 if kind == "static" else 4)
        h = 4.0 / min(nx, ny)
        body = rng.choice(["cylinder", "plate", "both"] if nx >= 128 else ["cylinder", "plate"])
        c = dict(kind=kind, nx=nx, ny=ny, levels=levels, h=h, body=body, Re=round(rng.uniform(50, 300), 1),
                 dt=round(0.2 * h, 6), steps=rng.randint(5, 20) if kind == "static" else rng.randint(2, 8))
        if kind == "static":
            c["precision"] = rng.choice(["fp64", "fp64", "fp64", "fp32", "mixed"])
            if c["precision"] != "fp64":
                c["steps"] = rng.randint(2, 6)
            c["grid"] = "moving" if c["precision"] == "fp64" and rng.random() < 0.2 else "fixed"
        return c
    if kind == "ensemble":
        precision = rng.choice(["fp64", "fp32"])
        return dict(kind=kind, count=rng.randint(3, 40), precision=precision,
                    steps=rng.randint(4, 16 if precision == "fp64" else 8))
    start = rng.choice(["previous", "extrapolated", "projected", "direct", "preconditioned", "preconditioned_extrapolated"])
    n = rng.choice([256, 512]) if start.startswith("precond") else _log_size(rng, 96, 512)
    products = rng.choice([0, 3]) if start.startswith("precond") else 0
    depth = rng.choice([4, 8, 16]) if start != "direct" else 1
    steps = rng.randint(1, 3) if start in ("previous", "extrapolated", "projected", "direct") else 2 * depth
    return dict(kind=kind, n=n, levels=rng.randint(2, 4), h=5.12 / n, k=round(rng.uniform(0.25, 0.85), 2),
                Re=round(rng.uniform(200, 600), 1), dt=round(0.2 * 5.12 / n, 6), steps=steps, start=start, depth=depth,
                products=products)


# --- geometry, built here so that run and exact see the same numbers ------------------------


def _circle(n, r, cx, cy):
    t = 2 * math.pi / n * np.arange(n)
    return np.column_stack([cx + r * np.cos(t), cy + r * np.sin(t)]), np.full(n, 2 * r * math.sin(math.pi / n))


def _line(n, ax, ay, bx, by):
    s = np.linspace(0.0, 1.0, n)
    return np.column_stack([ax + s * (bx - ax), ay + s * (by - ay)]), np.full(n, math.hypot(bx - ax, by - ay) / (n - 1))


def _plate(h, aoa, x=0.0, y=0.0):
    c, s = 0.5 * math.cos(aoa), 0.5 * math.sin(aoa)
    return _line(int(round(1.0 / h)) + 1, x - c, y + s, x + c, y - s)


def _flows(case, seed):
    """The flows of a case: a list of dicts of numbers and panel arrays."""
    rng = np.random.default_rng(seed)
    out = []
    if case["kind"] in ("static", "solve"):
        nx, ny, h = case["nx"], case["ny"], case["h"]
        aoa = math.radians(30.0 if case["kind"] == "static" else float(rng.uniform(0.0, 45.0)))
        cx, cy = (0.0, 0.0) if case["kind"] == "static" else (float(v) for v in rng.uniform(-0.1, 0.1, 2))
        panels = []
        if case["body"] in ("cylinder", "both"):
            panels.append(_circle(int(round(math.pi / h)), 0.5, cx, cy))
        if case["body"] == "plate":
            panels.append(_plate(h, aoa))
        if case["body"] == "both":
            panels.append(_plate(h, math.radians(15.0), 1.5, 0.3) if nx * h >= 4 else _plate(h, 0.0, 0.0, 1.2))
        # the body 40 % of the smaller side behind the inflow
        w, v = nx * h, ny * h
        out.append(dict(nx=nx, ny=ny, levels=case["levels"], h=h, xlim=(-0.4 * min(w, v), -0.4 * min(w, v) + w),
                        ylim=(-0.5 * v, 0.5 * v), Re=case["Re"], dt=case["dt"], panels=panels, moving=False,
                        grid=case.get("grid", "fixed"), noise=1e-3 if case["kind"] == "static" else 0.0))
    elif case["kind"] == "moving":
        n, h = case["n"], case["h"]
        s = n * h
        out.append(dict(nx=n, ny=n, levels=case["levels"], h=h, xlim=(-0.3 * s, -0.3 * s + s), ylim=(-0.5 * s, 0.5 * s),
                        Re=case["Re"], dt=case["dt"], panels=[_line(int(round(1.0 / h)) + 1, -0.5, 0.0, 0.5, 0.0)],
                        moving=True, grid="fixed", noise=1e-3, k=case["k"]))
    else:  # ensembles of {256, 384, 512} x 256 cells, cylinders or plates
        h, ny = 0.01, 256
        shapes = np.random.default_rng(case["count"])  # widths and bodies go with the case, the rest with the seed
        for _ in range(case["count"]):
            nx = int(shapes.choice([256, 384, 512]))
            Re = float(rng.uniform(50.0, 300.0))
            if shapes.uniform() < 0.5:
                D = float(shapes.uniform(0.5, 1.5))
                panels = [_circle(int(round(math.pi * D / h)), D / 2, 0.0, 0.0)]
            else:
                panels = [_plate(h, math.radians(float(rng.uniform(0.0, 45.0))))]
            v = ny * h
            out.append(dict(nx=nx, ny=ny, levels=3, h=h, xlim=(-0.4 * v, -0.4 * v + nx * h), ylim=(-0.5 * v, 0.5 * v),
                            Re=Re, dt=0.002, panels=panels, moving=False, grid="fixed", noise=1e-3))
    for f in out:  # vorticity noise, one stream for all levels
        f["noise_seed"] = int(rng.integers(1 << 31))
    return out


def _noise(f):
    rng = np.random.default_rng(f["noise_seed"])
    ng = (f["nx"] - 1) * (f["ny"] - 1)
    return [rng.standard_normal(ng) * (f["noise"] * (f["h"] * 2 ** lev) ** 2) for lev in range(f["levels"])]


def _grid_motion(t):
    """center, velocity, angle, angular velocity of the moving grid"""
    return (-1.0, 0.0), (0.0, 0.2 * math.cos(t)), 0.1 * math.sin(t), 0.1 * math.cos(t)


def _plate_motion(k, t):
    """position, velocity, angle, angular velocity of the pitching and plunging plate"""
    w, th = 2 * k, math.radians(30.0)
    return ((0.0, 0.25 * math.sin(w * t)), (0.0, 0.25 * w * math.cos(w * t)), -th * math.sin(w * t),
            -th * w * math.cos(w * t))


def _problem(f):
    motion = ib.MovingGrid(lambda t: ib.GridVelocity(*_grid_motion(t))) if f["grid"] == "moving" else None
    fluid = ib.Fluid(grid=ib.fluid_grid(h=f["h"], xlims=f["xlim"], ylims=f["ylim"], nlevel=f["levels"]), Re=f["Re"],
                     freestream_vel=lambda t: (1.0, 0.0), grid_motion=motion)
    bodies = {}
    for i, (xb, ds) in enumerate(f["panels"]):
        p = ib.Panels(xb, ds)
        bodies["b%d" % i] = (ib.MovingRigidBody(lambda t: ib.RigidBodyTransform(*_plate_motion(f["k"], t)), p)
                             if f["moving"] else ib.StaticBody(p))
    return ib.Problem(fluid=fluid, bodies=ib.Bodies(bodies), scheme=ib.CNAB(dt=f["dt"]))


def _state(f):
    st = ib.State(_problem(f))
    if f["noise"]:
        for lev, g in enumerate(_noise(f)):
            st.Gamma[:, lev] = g
    return st


# --- prepare and run -------------------------------------------------------------------------


def prepare(case, seed):
    if case["kind"] == "poisson":
        g = torch.Generator(device="cuda").manual_seed(seed)
        b = torch.randn(case["ny"] - 1, case["nx"] - 1, generator=g, device="cuda", dtype=torch.float64)
        return dict(case=case, b=b, x=torch.empty_like(b), lib=ib._abi.load())
    flows = _flows(case, seed)
    if case["kind"] == "solve":
        return dict(case=case, prob=_problem(flows[0]))
    if case["kind"] == "ensemble":
        solvers = [ib.GpuCnabSolver(_state(f), precision=case["precision"]) for f in flows]
        return dict(case=case, ens=ib.Ensemble(solvers))
    if case["kind"] == "static":
        return dict(case=case, solver=ib.create_solver(_state(flows[0]), precision=case["precision"]))
    s = ib.create_solver(_state(flows[0]))
    if case["start"] != "previous":
        s.set_warm_start(None, mode=case["start"], depth=case["depth"])
        if case["products"]:
            s.set_rebuild_transform(case["products"])
    return dict(case=case, solver=s)


def run(state):
    case = state["case"]
    if case["kind"] == "poisson":
        b, x = state["b"], state["x"]
        rc = state["lib"].ibpm_lap_inv_noalloc(case["nx"], case["ny"], ctypes.c_void_p(b.data_ptr()),
                                               ctypes.c_void_p(x.data_ptr()),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError("ibpm_lap_inv_noalloc failed")
        return x
    if case["kind"] == "ensemble":
        ens = state["ens"]
        ens.advance_(case["steps"])
        vort = [s.vorticity(1) for s in ens.solvers]
        if case["precision"] != "fp64":
            return {"vorticity": [v.astype(np.float32) for v in vort]}
        return {"forces": np.concatenate([s.state.fb for s in ens.solvers]), "vorticity": vort}
    if case["kind"] == "solve":
        solver = ib.solve(state["prob"], t=(case["steps"] - 1) * case["dt"])
        forces = solver.state.fb.copy()
    else:
        solver, forces = state["solver"], []
        for _ in range(case["steps"]):
            ib.advance_(solver)
            forces.append(solver.state.fb.copy())
        forces = np.stack(forces)
    vort = [solver.vorticity(lev + 1) for lev in range(case["levels"])]
    if case.get("precision", "fp64") != "fp64":
        return {"vorticity": [v.astype(np.float32) for v in vort]}
    return {"forces": forces, "vorticity": vort}


def work(case):
    """Bytes and operations of one pass.  A step reads Gamma, q and the previous
    nonlinear term and writes Gamma, psi, q and the nonlinear term once per
    level; its transforms are six 2D sine transforms a level (trial solve, and
    vort2flux twice) and two for the correction, at 2.5 n log2 n each line."""
    if case["kind"] == "poisson":
        n = (case["nx"] - 1) * (case["ny"] - 1)
        return {"bytes": 16 * n, "flops": 5 * n * math.log2(case["nx"] * case["ny"])}
    size = 8 if case.get("precision", "fp64") == "fp64" else 4
    nbytes = flops = 0.0
    for f in _flows(case, 0):
        g, q = (f["nx"] - 1) * (f["ny"] - 1), (f["nx"] + 1) * f["ny"] + f["nx"] * (f["ny"] + 1)
        m = 2 * sum(len(p[0]) for p in f["panels"])
        per = size * f["levels"] * (2 * q + 5 * g) + 8 * m * m
        ops = f["levels"] * (6 * 2.5 * g * math.log2(f["nx"] * f["ny"]) + 60 * g) + 2 * m * m
        nbytes += case["steps"] * per + 8 * g * (1 if case["kind"] == "ensemble" else f["levels"])
        flops += case["steps"] * ops
    return {"bytes": nbytes, "flops": flops}


# --- the method in plain torch, float64 ------------------------------------------------------


def _delta(r):
    """Yang et al. (JCP 2009) smoothed three-point delta, r in cells (numpy)."""
    r = np.abs(r)
    r2, r3, r4 = r * r, r ** 3, r ** 4
    with np.errstate(invalid="ignore"):
        a = np.arcsin(0.5 * math.sqrt(3.0) * (2 * r - 1))
        s = np.sqrt(1 - 12 * r2 + 12 * r)
        v1 = (4.166666667e-2 * r4 + (-0.1388888889 + 3.472222222e-2 * s) * r3
              + (-7.121664902e-2 - 5.208333333e-2 * s + 0.2405626122 * a) * r2
              + (-0.2405626122 * a - 0.3792313933 + 0.1012731481 * s) * r
              + 8.0187537413e-2 * a - 4.195601852e-2 * s + 0.6485698427)
        a = np.arcsin(0.5 * math.sqrt(3.0) * (-3 + 2 * r))
        s = np.sqrt(-23 + 36 * r - 12 * r2)
        v2 = (-6.25e-2 * r4 + (0.4861111111 - 1.736111111e-2 * s) * r3
              + (-1.143175026 + 7.8125e-2 * s - 0.1202813061 * a) * r2
              + (0.8751991178 + 0.3608439183 * a - 0.1548032407 * s) * r - 0.2806563809 * a + 8.22848104e-3
              + 0.1150173611 * s)
        a = np.arcsin(0.5 * math.sqrt(3.0) * (2 * r - 5))
        s = np.sqrt(-71 - 12 * r2 + 60 * r)
        v3 = (2.083333333e-2 * r4 + (3.472222222e-3 * s - 0.2638888889) * r3
              + (1.214391675 - 2.604166667e-2 * s + 2.405626122e-2 * a) * r2
              + (-0.1202813061 * a - 2.449273192 + 7.262731481e-2 * s) * r + 0.1523563211 * a + 1.843201677
              - 7.306134259e-2 * s)
    return np.where(r <= 1, v1, np.where(r <= 2, v2, np.where(r <= 3, v3, 0.0)))


class _Exact:
    """One flow stepped in plain torch; fields are (..., nx-1, ny-1), x first."""

    def __init__(self, f):
        self.f, self.dev = f, "cuda"
        nx, ny, self.L, self.h, self.dt, self.Re = f["nx"], f["ny"], f["levels"], f["h"], f["dt"], f["Re"]
        self.nx, self.ny = nx, ny
        k = lambda n: torch.arange(1, n, dtype=torch.float64, device=self.dev)  # noqa: E731
        # sine matrices from exact integer phases mod 2 n
        sine = lambda n: torch.sin(math.pi / n * ((torch.arange(1, n)[:, None] * torch.arange(1, n)) % (2 * n)).double()).to(self.dev)  # noqa: E731
        self.Sx, self.Sy = sine(nx), sine(ny)
        self.lam = -2 * (torch.cos(math.pi * k(nx) / nx)[:, None] + torch.cos(math.pi * k(ny) / ny)[None, :] - 2)
        self.G = torch.stack([torch.from_numpy(g.reshape(ny - 1, nx - 1).T.copy()) for g in _noise(f)]).to(self.dev)
        self.qx = torch.zeros(self.L, nx + 1, ny, dtype=torch.float64, device=self.dev)
        self.qy = torch.zeros(self.L, nx, ny + 1, dtype=torch.float64, device=self.dev)
        self.N2 = torch.zeros_like(self.G)
        self.ref = np.concatenate([p[0] for p in f["panels"]])
        self.t = 0.0
        if not f["moving"]:
            self.place(self.ref, np.zeros_like(self.ref))

    def hc(self, lev):
        return self.h * 2.0 ** lev

    def solve(self, den, b):
        """S(S(b) / den) / (4 nx ny) with S the unnormalised DST-I (2 sin) in both directions"""
        t = self.Sx @ b @ self.Sy / den
        return self.Sx @ t @ self.Sy * (4.0 / (self.nx * self.ny))

    def implicit(self, lev):
        return 1 + self.lam * (self.dt / (2 * self.Re * self.hc(lev) ** 2))

    def place(self, xb, ub):
        x0, y0, h = float(self.f["xlim"][0]), float(self.f["ylim"][0]), self.h
        ix = np.rint((xb[:, 0] - x0) / h + 1 - 0.25).astype(int)
        iy = np.rint((xb[:, 1] - y0) / h + 1 - 0.25).astype(int)
        o = np.arange(-3, 4)
        X, Y = x0 + h * ((ix[:, None] + o) - 1), y0 + h * ((iy[:, None] + o) - 1)
        bx, by = xb[:, :1], xb[:, 1:]
        wx = _delta((X - bx) / h)[:, :, None] * _delta((Y + h / 2 - by) / h)[:, None, :]
        wy = _delta((X + h / 2 - bx) / h)[:, :, None] * _delta((Y - by) / h)[:, None, :]
        I, J = (ix[:, None] + o - 1)[:, :, None], (iy[:, None] + o - 1)[:, None, :]
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        self.wx, self.wy = put(wx).flatten(1), put(wy).flatten(1)
        self.ku, self.kv = put(I * self.ny + J).flatten(1), put(I * (self.ny + 1) + J).flatten(1)
        self.ub = put(ub)
        self.B = None

    def E(self, qx, qy):
        """(..., nx+1, ny), (..., nx, ny+1) -> (..., 2 np)"""
        fx = (qx.flatten(-2)[..., self.ku] * self.wx).sum(-1)
        fy = (qy.flatten(-2)[..., self.kv] * self.wy).sum(-1)
        return torch.cat([fx, fy], -1)

    def ET_rot(self, F):
        """rot of E^T F, F (..., 2 np)"""
        n = self.wx.shape[0]
        lead = F.shape[:-1]
        qx = torch.zeros(*lead, (self.nx + 1) * self.ny, dtype=torch.float64, device=self.dev)
        qy = torch.zeros(*lead, self.nx * (self.ny + 1), dtype=torch.float64, device=self.dev)
        qx.index_add_(-1, self.ku.flatten(), (F[..., :n, None] * self.wx).flatten(-2))
        qy.index_add_(-1, self.kv.flatten(), (F[..., n:, None] * self.wy).flatten(-2))
        return self.rot(qx.view(*lead, self.nx + 1, self.ny), qy.view(*lead, self.nx, self.ny + 1))

    @staticmethod
    def rot(qx, qy):
        return qx[..., 1:-1, :-1] - qx[..., 1:-1, 1:] + qy[..., 1:, 1:-1] - qy[..., :-1, 1:-1]

    def bc(self, r):
        """Boundary values from the coarser level's field: bottom, top (nx+1), left, right (ny+1)."""
        nx, ny = self.nx, self.ny

        def fine(v):
            out = torch.zeros(*v.shape[:-1], 2 * v.shape[-1] - 1, dtype=torch.float64, device=self.dev)
            out[..., ::2] = v
            out[..., 1::2] = 0.5 * (v[..., 1:] + v[..., :-1])
            return out

        xs, ys = slice(nx // 4 - 1, nx // 4 + nx // 2), slice(ny // 4 - 1, ny // 4 + ny // 2)
        return (fine(r[..., xs, ny // 4 - 1]), fine(r[..., xs, 3 * ny // 4 - 1]), fine(r[..., nx // 4 - 1, ys]),
                fine(r[..., 3 * nx // 4 - 1, ys]))

    def add_bc(self, r, bc, fac):
        r = r.clone()
        r[..., :, 0] += fac * bc[0][..., 1:-1]
        r[..., :, -1] += fac * bc[1][..., 1:-1]
        r[..., 0, :] += fac * bc[2][..., 1:-1]
        r[..., -1, :] += fac * bc[3][..., 1:-1]
        return r

    def framed(self, r, bc):
        """r with its boundary values around it: (..., nx+1, ny+1) grid vertices"""
        p = torch.zeros(*r.shape[:-2], self.nx + 1, self.ny + 1, dtype=torch.float64, device=self.dev)
        if bc is not None:
            p[..., :, 0], p[..., :, -1], p[..., 0, :], p[..., -1, :] = bc
        p[..., 1:-1, 1:-1] = r
        return p

    def coarsify(self, G):
        """Levels 2.. take the finer level's vorticity in their central block, in place; G (..., L, nx-1, ny-1)."""
        nx, ny = self.nx, self.ny
        for lev in range(1, self.L):
            F = G[..., lev - 1, :, :]
            # 0-based first centre on the fine level, first point on the coarse one, and the counts
            i0, ic, ni = 1, nx // 2 - nx // 4, min((nx - 4) // 2 + 1, 2 * (nx // 4) - 1)
            j0, jc, nj = 1, ny // 2 - ny // 4, min((ny - 4) // 2 + 1, 2 * (ny // 4) - 1)
            at = lambda a, b: F[..., i0 + a: i0 + a + 2 * ni - 1: 2, j0 + b: j0 + b + 2 * nj - 1: 2]  # noqa: E731
            G[..., lev, ic: ic + ni, jc: jc + nj] = (at(0, 0) + 0.5 * (at(1, 0) + at(0, 1) + at(-1, 0) + at(0, -1))
                                                    + 0.25 * (at(1, 1) + at(1, -1) + at(-1, -1) + at(-1, 1)))

    def flux(self, G, every):
        """vort2flux: psi and flux of every level, or the flux of level 1; G is coarsified in place."""
        self.coarsify(G)
        bc, out = None, []
        for lev in range(self.L - 1, -1, -1):
            r = G[..., lev, :, :]
            psi = self.solve(self.lam, r if bc is None else self.add_bc(r, bc, 1.0))
            if every or lev == 0:
                p = self.framed(psi, bc)
                out.append((p[..., :, 1:] - p[..., :, :-1], p[..., :-1, :] - p[..., 1:, :]))
            bc = self.bc(psi)
        return out[::-1]

    def Bcols(self, F):
        G = torch.zeros(*F.shape[:-1], self.L, self.nx - 1, self.ny - 1, dtype=torch.float64, device=self.dev)
        G[..., 0, :, :] = self.solve(self.implicit(0), self.ET_rot(F))
        return self.E(*self.flux(G, False)[0])

    def base(self, lev, t):
        """base flux of a level: x faces, y faces"""
        hc, nx, ny = self.hc(lev), self.nx, self.ny
        if self.f["grid"] != "moving":
            return hc * 1.0, 0.0
        (cx, cy), (ux, uy), th, om = _grid_motion(t)
        c, s = math.cos(th), math.sin(th)
        x0 = self.f["xlim"][0] + nx * (self.h - hc) / 2
        y0 = self.f["ylim"][0] + ny * (self.h - hc) / 2
        ar = lambda n: torch.arange(n, dtype=torch.float64, device=self.dev)  # noqa: E731

        def wind(x, y):
            dx, dy = (x - cx)[:, None], (y - cy)[None, :]
            return 1.0 - ux - om * (-s * dx - c * dy), -uy - om * (c * dx - s * dy)

        wx, wy = wind(x0 + hc * ar(nx + 1), y0 + hc / 2 + hc * ar(ny))
        vx, vy = wind(x0 + hc / 2 + hc * ar(nx), y0 + hc * ar(ny + 1))
        return hc * (c * wx + s * wy), hc * (-s * vx + c * vy)

    def nonlinear(self, lev, q0, bc):
        qx, qy = self.qx[lev] + q0[0], self.qy[lev] + q0[1]
        ax = torch.zeros(self.nx + 1, self.ny + 1, dtype=torch.float64, device=self.dev)  # average x flux at vertices
        ay = torch.zeros_like(ax)
        ax[:, 1:-1] = (qx[:, 1:] + qx[:, :-1]) / 2
        ay[1:-1, :] = (qy[1:, :] + qy[:-1, :]) / 2
        # the average flux is along the faces of the level, so the outermost rows and columns take its own values
        g = self.framed(self.G[lev], None if bc is None else [0.25 * v for v in bc])
        px, py = ay * g, ax * g
        fx = (px[:, 1:] + px[:, :-1]) / 2
        fy = -(py[1:, :] + py[:-1, :]) / 2
        return self.rot(fx, fy) / self.hc(lev) ** 2

    def step(self):
        f, t = self.f, self.t
        if f["moving"]:
            (px, py), (vx, vy), a, om = _plate_motion(f["k"], t)
            c, s, r = math.cos(a), math.sin(a), self.ref
            self.place(np.column_stack([px + (c * r[:, 0] - s * r[:, 1]), py + (s * r[:, 0] + c * r[:, 1])]),
                       np.column_stack([vx + om * (-s * r[:, 0] - c * r[:, 1]), vy + om * (c * r[:, 0] - s * r[:, 1])]))
        if self.B is None:
            n = 2 * self.wx.shape[0]
            eye = torch.eye(n, dtype=torch.float64, device=self.dev)
            w = max(1, int((2 << 30) / (8 * self.L * self.nx * self.ny)))
            self.B = torch.cat([self.Bcols(eye[k: k + w]) for k in range(0, n, w)]).T
            self.lu = torch.linalg.lu_factor(self.B)
        new, N1 = torch.empty_like(self.G), torch.empty_like(self.G)
        for lev in range(self.L):
            hc = self.hc(lev)
            bc = self.bc(self.G[lev + 1]) if lev + 1 < self.L else None
            N1[lev] = self.nonlinear(lev, self.base(lev, t), bc)
            rhs = self.solve(1 / (1 - self.lam * (self.dt / (2 * self.Re * hc ** 2))), self.G[lev])
            rhs = rhs + self.dt * (1.5 * N1[lev] - 0.5 * self.N2[lev])
            if bc is not None:
                rhs = self.add_bc(rhs, bc, 0.25 * self.dt / (self.Re * hc ** 2))
            new[lev] = self.solve(self.implicit(lev), rhs)
        self.N2 = N1
        q1 = self.flux(new, False)[0]
        q0 = self.base(0, t)
        F = self.E(q1[0] + q0[0], q1[1] + q0[1]) - self.ub.T.flatten() * self.h
        F = torch.linalg.lu_solve(*self.lu, F[:, None])[:, 0]
        new[0] -= self.solve(self.implicit(0), self.ET_rot(F))
        self.G = new
        for lev, (x, y) in enumerate(self.flux(self.G, True)):
            self.qx[lev], self.qy[lev] = x, y
        self.t += self.dt
        return (F * self.h / self.dt).view(2, -1).T

    def vorticity(self, lev):
        return (self.G[lev] / self.hc(lev) ** 2).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "poisson":
        b = prepare(case, seed)["b"].T
        nx, ny = case["nx"], case["ny"]
        e = _Exact(dict(nx=nx, ny=ny, levels=1, h=1.0, dt=1.0, Re=1.0, panels=[(np.zeros((0, 2)), None)], moving=True,
                        noise=0.0, noise_seed=0))
        return e.solve(e.lam, b).T.contiguous()
    flows = _flows(case, seed)
    if case["kind"] == "ensemble":
        vort, forces, known = [], [], len(flows) <= 20 or case["precision"] != "fp64"
        for i, f in enumerate(flows):
            if i >= (20 if case["precision"] == "fp64" else 12):  # about 1 s a case
                vort.append(None)
                continue
            e = _Exact(f)
            for _ in range(case["steps"]):
                fb = e.step()
            forces.append(fb.cpu().numpy())
            vort.append(e.vorticity(0))
        if case["precision"] != "fp64":
            return {"vorticity": vort}
        return {"forces": np.concatenate(forces) if known else None, "vorticity": vort}
    e, forces = _Exact(flows[0]), []
    for _ in range(case["steps"]):
        forces.append(e.step().cpu().numpy())
    vort = [e.vorticity(lev) for lev in range(case["levels"])]
    if case.get("precision", "fp64") != "fp64":
        return {"vorticity": vort}
    return {"forces": forces[-1] if case["kind"] == "solve" else np.stack(forces), "vorticity": vort}
