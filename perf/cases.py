"""Performance cases: the work that programs have this package do, through its public entry points.

Operators and whole solves on one grid (the reference's `op!(out, in, cache)` calls and the `solve` of its
Poisson, Stokes and heat problems), and the batched solver.  `exact` restates each in FP64 with plain torch.
Grids span [-2, 2]^2-like boxes (h = 4 / nx); bodies are ellipses whose centre, aspect and angle come from the
seed, with a fixed number of points per body.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "immersedlayers.jl_gb300"))

import immersedlayers as il  # noqa: E402
from immersedlayers import learned as LN  # noqa: E402
from immersedlayers import workloads as W  # noqa: E402
from immersedlayers.batch import DIRICHLET, BatchProblemSpec, BatchSolver, PackedBatch  # noqa: E402

DT = {"float64": torch.float64, "float32": torch.float32}
BATCH_SIZES = (128, 192, 256, 384, 512)
TOL = 1e-12         # the reference solves its Schur systems by dense LU in FP64
BATCH_TOL = 1e-8    # the batched solver's published residual


def listed():
    return [
        # a layer chain on the reference's unit-test grid (h = 0.04, ds = 1.4 h): latency and launches
        {"name": "layer_106_f64", "op": "layer", "dtype": "float64", "nx": 106, "ny": 106, "bodies": 1, "pts": 112},
        # the same chain at the operators-at-scale size, single precision (points 0.25 h apart)
        {"name": "layer_1024_f32", "op": "layer", "dtype": "float32", "nx": 1024, "ny": 1024, "bodies": 3,
         "pts": 4095},
        # staggered-grid calculus and convective terms at the largest grid of the stencil benchmark, ragged rows
        {"name": "calculus_4096_f32", "op": "calculus", "dtype": "float32", "nx": 4096, "ny": 4001},
        # a large unbounded-domain inverse Laplacian (the Stokes configuration's grid)
        {"name": "invlap_2048_f64", "op": "invlap", "dtype": "float64", "nx": 2048, "ny": 2048},
        # Helmholtz reconstruction of a vector field, an odd rectangular grid
        {"name": "helmholtz_901x607_f64", "op": "helmholtz", "dtype": "float64", "nx": 901, "ny": 607, "bodies": 2,
         "pts": 500},
        # the plain Dirichlet configuration, solved again and again on a kept cache
        {"name": "dirichlet_206_f64", "op": "dirichlet", "dtype": "float64", "nx": 206, "ny": 206, "bodies": 1,
         "pts": 157},
        # the literate Neumann problem (potential and streamfunction) on the reference's printed grid
        {"name": "neumann_406_f64", "op": "neumann", "dtype": "float64", "nx": 406, "ny": 406, "bodies": 1,
         "pts": 448},
        # moving bodies: new points, then a Dirichlet solve that needs a new Schur complement
        {"name": "moving_512_f64", "op": "moving", "dtype": "float64", "nx": 512, "ny": 512, "bodies": 3,
         "pts": 696},
        # heat conduction at ds = 1.4 h, marched ten steps
        {"name": "heat_1024_f64", "op": "heat", "dtype": "float64", "nx": 1024, "ny": 1024, "bodies": 3, "pts": 726,
         "steps": 10},
        # the Stokes example's grid, two bodies of its point count
        {"name": "stokes_406_f64", "op": "stokes", "dtype": "float64", "nx": 406, "ny": 406, "bodies": 2,
         "pts": 428},
        # a batch of independent problems, geometry kept, solved with the default solver
        {"name": "batch_solve_64_f32", "op": "batch", "dtype": "float32", "problems": 64, "setup": False},
        # the same from packed host arrays: set-up, preconditioners and the solve
        {"name": "batch_setup_64_f32", "op": "batch", "dtype": "float32", "problems": 64, "setup": True},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    op = rng.choice(("layer", "calculus", "invlap", "helmholtz", "dirichlet", "neumann", "moving", "heat", "stokes",
                     "batch"))
    if op == "batch":
        return {"op": op, "dtype": "float32", "problems": rng.randint(5, 63), "setup": rng.random() < 0.5}
    top = {"layer": 1024, "calculus": 4000, "invlap": 2000, "helmholtz": 800, "dirichlet": 500, "neumann": 400,
           "moving": 500, "heat": 1000, "stokes": 300}[op]
    nx = _log(rng, 100, top)
    ny = max(96, min(top, int(nx * rng.uniform(0.7, 1.1))))
    c = {"op": op, "dtype": rng.choice(("float64", "float32")) if op in ("layer", "calculus", "invlap") else "float64",
         "nx": nx, "ny": ny}
    if op in ("calculus", "invlap"):
        return c
    c["bodies"] = rng.randint(1, 2 if op == "stokes" else 3)
    # ds from 1.4 h upwards for the solves; the transfers also take denser points
    per_body = rng.uniform(0.2, 0.42) * min(nx, ny) * (rng.uniform(1.0, 5.0) if op == "layer" else 1.0)
    c["pts"] = c["bodies"] * max(16, int(per_body))
    if op == "heat":
        c["steps"] = rng.randint(3, 10)
    return c


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _bodies(case, seed):
    """`bodies` ellipses with `pts` points in all, each in its own third of the box (fewer bodies: larger ones)."""
    rng = np.random.default_rng([seed, 11])
    nb, h = case["bodies"], 4.0 / case["nx"]
    wx, wy = 2.0, 2.0 * case["ny"] / case["nx"]
    n = case["pts"] // nb
    # semi-axes from the perimeter that keeps the points at least 1.4 h apart where the box has room for it
    cell = min(wx, wy) * (0.62 if nb == 1 else 0.27)
    dense = n * 1.4 * h / (2 * math.pi) > cell
    bl = il.BodyList()
    turn = rng.uniform(0, 2 * math.pi)
    for b in range(nb):
        a = cell if dense else n * 1.42 * h / (2 * math.pi) * rng.uniform(1.0, 1.05)
        e = rng.uniform(0.75, 1.0)
        cx = cy = 0.0
        if nb > 1:
            t = turn + 2 * math.pi * b / nb
            d = 0.54 * min(wx, wy)
            cx, cy = d * math.cos(t), d * math.sin(t)
        cx += rng.uniform(-1.5, 1.5) * h
        cy += rng.uniform(-1.5, 1.5) * h
        # same perimeter for every aspect (Ramanujan)
        k = ((1 - e) / (1 + e)) ** 2
        per = (1 + e) / 2 * (1 + 3 * k / (10 + math.sqrt(4 - 3 * k)))
        bl.append(il.ellipse(a / per, a * e / per, n=n + (case["pts"] - nb * n if b == 0 else 0), center=(cx, cy),
                             angle=rng.uniform(0, math.pi)))
    return bl


def _grid(case):
    return il.PhysicalGrid.from_cells(case["nx"], 4.0 / case["nx"], ny=case["ny"])


def _surface(bl, seed, k=1):
    """k columns of smooth surface data with a little noise on top."""
    rng = np.random.default_rng([seed, 12])
    return [W.fourier_surface_data(bl, rng) for _ in range(k)]


def _dev(a, dtype):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64).to("cuda").to(dtype)


def _smooth(n1, n2, seed, k, dtype):
    """A random field: a few waves plus white noise, made on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(1000 * seed + k)
    x = torch.linspace(-1, 1, n1, dtype=torch.float64, device="cuda")
    y = torch.linspace(-1, 1, n2, dtype=torch.float64, device="cuda")
    p = torch.rand(6, generator=g, device="cuda", dtype=torch.float64) * 6.0
    f = torch.sin(p[0] * x + p[1])[None, :] * torch.cos(p[2] * y + p[3])[:, None]
    f = f + 0.1 * torch.randn(n2, n1, generator=g, device="cuda", dtype=torch.float32)
    return f.to(dtype).reshape(-1)


_SHAPES = {"P": (0, 0), "D": (1, 1), "U": (1, 0), "V": (0, 1)}


def _shape(case, pc):
    dx, dy = _SHAPES[pc]
    return case["nx"] - 1 + dx, case["ny"] - 1 + dy


def _field(case, seed, pcs, k, dtype):
    return torch.cat([_smooth(*_shape(case, pc), seed, k + i, dtype) for i, pc in enumerate(pcs)])


def _batch_problem(i):
    """Grid size, bodies and points of problem i: the sizes and mean point counts of the batched configuration."""
    n, nb = BATCH_SIZES[(3 * i + i // 5) % 5], 1 + (i // 2) % 3
    return {"nx": n, "ny": n, "bodies": nb, "pts": nb * int(n * (0.24 + 0.18 * (7 * i % 8) / 7))}


def _batch_specs(case, seed):
    specs = []
    for i in range(case["problems"]):
        p = _batch_problem(i)
        bl = _bodies(p, 1000 * seed + i)
        specs.append(BatchProblemSpec(p["nx"], 4.0 / p["nx"], bl, i % 2, _surface(bl, 1000 * seed + i)[0]))
    return specs


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, op, dt = case, case["op"], DT[case["dtype"]]
    if op == "batch":
        s.specs = _batch_specs(case, seed)
        s.packed = PackedBatch(s.specs)
        s.net = LN.LearnedPreconditioner.load(LN.BATCHED_WEIGHTS[DIRICHLET])
        if not case["setup"]:
            s.solver = _batch_solver(s)
            s.solver.set_rhs_operator(True)   # a program that solves the same geometry many times
            s.fp, s.fm = s.solver.surface_data()
            s.f = torch.empty(s.solver.total_cells, dtype=dt, device="cuda")
            s.s = torch.empty(s.solver.total_points, dtype=dt, device="cuda")
        else:
            s.fp = _dev(np.concatenate([p.fplus for p in s.specs]), dt)
            s.fm = torch.zeros_like(s.fp)
        return s
    s.grid = _grid(case)
    if op in ("calculus", "invlap"):
        s.cache = il.SurfaceScalarCache(None, s.grid, dtype=dt)
        if op == "invlap":
            s.w = il.NodesPrimal(s.grid, _field(case, seed, "P", 0, dt))
            s.out = il.NodesPrimal.zeros(s.grid, dt)
            return s
        s.p = il.NodesPrimal(s.grid, _field(case, seed, "P", 0, dt))
        s.d = il.NodesDual(s.grid, _field(case, seed, "D", 1, dt))
        s.v = il.EdgesPrimal(s.grid, _field(case, seed, "UV", 2, dt))
        s.o = [t.zeros(s.grid, dt) for t in (il.EdgesPrimal, il.NodesPrimal, il.EdgesPrimal, il.NodesDual,
                                             il.NodesPrimal, il.EdgesPrimal, il.EdgesPrimal)]
        return s
    bl = s.bl = _bodies(case, seed)
    if op == "layer":
        s.cache = il.SurfaceScalarCache(bl, s.grid, dtype=dt)
        s.f = il.ScalarData(_dev(_surface(bl, seed)[0], dt))
        s.theta, s.w = il.zeros_grid(s.cache), il.zeros_grid(s.cache)
        s.g = il.zeros_surface(s.cache)
    elif op == "helmholtz":
        s.cache = il.SurfaceVectorCache(bl, s.grid, dtype=dt)
        s.curlv = il.NodesDual(s.grid, _field(case, seed, "D", 0, dt))
        s.divv = il.NodesPrimal(s.grid, _field(case, seed, "P", 1, dt))
        s.dv = il.VectorData(_dev(np.concatenate(_surface(bl, seed, 2)), dt))
        s.v = il.EdgesPrimal.zeros(s.grid, dt)
        s.vf = il.VectorFieldCache(s.cache)
    elif op in ("dirichlet", "neumann"):
        s.cache = il.SurfaceScalarCache(bl, s.grid, dtype=dt)
        s.plus, s.minus = (il.ScalarData(_dev(a, dt)) for a in _surface(bl, seed, 2))
    elif op == "moving":
        start = _bodies(case, seed + 500)
        s.cache = il.SurfaceScalarCache(start, s.grid, dtype=dt)
        s.points = [_dev(a, torch.float64) for a in (bl.x, bl.y, bl.nx, bl.ny, bl.ds)]
        s.plus, s.minus = (il.ScalarData(_dev(a, dt)) for a in _surface(bl, seed, 2))
    elif op == "heat":
        h = s.grid.h
        tb = _surface(bl, seed, 2)
        prob = il.DirichletHeatConductionProblem(
            g=s.grid, bodies=bl, dtype=dt, phys_params={"diffusivity": 1.0, "Fourier": 0.5},
            bc={"exterior": lambda c, p: tb[0], "interior": lambda c, p: tb[1]})
        system = il.construct_system(prob)
        s.T0 = _field(case, seed, "P", 0, dt)
        s.integ = il.init(il.init_sol(system, s.T0), (0.0, 1.0), system, dt=0.5 * h * h, tol=TOL)
    elif op == "stokes":
        s.cache = il.SurfaceVectorCache(bl, s.grid, dtype=dt)
        s.plus, s.minus = (il.VectorData(_dev(a, dt)) for a in _velocities(bl, seed))
    return s


def _velocities(bl, seed):
    """Rigid motion of every body outside, its rotation alone inside."""
    rng = np.random.default_rng([seed, 13])
    plus, minus, fi = np.zeros(2 * len(bl)), np.zeros(2 * len(bl)), bl.firstindices()
    for b in range(len(bl.bodies)):
        k = slice(fi[b], fi[b + 1])
        x, y = bl.x[k] - bl.x[k].mean(), bl.y[k] - bl.y[k].mean()
        ux, uy, om = rng.standard_normal(3)
        for v, t in ((plus, 1.0), (minus, 0.0)):
            v[k] = t * ux - om * y
            v[len(bl) + fi[b]:len(bl) + fi[b + 1]] = t * uy + om * x
    return plus, minus


def _batch_solver(s):
    b = BatchSolver(s.specs, dtype=DT[s.case["dtype"]], packed=s.packed)
    b.set_precond("bjacobi", 64)
    b.set_learned(s.net, kinds=(DIRICHLET,))
    b.set_coarse(True)
    return b


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def run(s):
    op = s.case["op"]
    if op == "layer":      # f* = L^-1 D_s [f] and its surface values
        il.surface_divergence_(s.theta, s.f, s.cache)
        il.inverse_laplacian_(s.w, s.theta, s.cache)
        il.interpolate_(s.g, s.w, s.cache)
        return {"theta": s.theta.data, "w": s.w.data, "g": s.g.data}
    if op == "calculus":
        c, o = s.cache, s.o
        il.grad_(o[0], s.p, c)
        il.divergence_(o[1], s.v, c)
        il.curl_(o[2], s.d, c)
        il.curl_(o[3], s.v, c)
        il.laplacian_(o[4], s.p, c)
        il.convective_derivative_(o[5], s.v, c)
        il.w_cross_v_(o[6], s.d, s.v, c)
        return [a.data for a in o]
    if op == "invlap":
        return il.inverse_laplacian_(s.out, s.w, s.cache).data
    if op == "helmholtz":
        return il.vecfield_helmholtz_(s.v, s.curlv, s.divv, s.dv, (0.3, -0.2), s.cache, s.vf).data
    if op == "dirichlet":
        f, x, _ = il.solve_dirichlet(s.cache, s.plus, s.minus, tol=TOL, maxiter=20000)
        return {"f": f.data, "s": x.data}
    if op == "neumann":
        f, df, psi, dpsi, _ = il.solve_neumann_full(s.cache, s.plus, s.minus, tol=TOL, maxiter=20000)
        return {"f": f.data, "df": df.data, "psi": psi.data, "dpsi": dpsi.data}
    if op == "moving":
        s.cache.update_points_(*s.points)
        f, x, _ = il.solve_dirichlet(s.cache, s.plus, s.minus, tol=TOL, maxiter=20000)
        return {"f": f.data, "s": x.data}
    if op == "heat":
        s.integ.u.state.data.copy_(s.T0)
        s.integ.advance(s.case["steps"])
        return {"T": s.integ.u.state.data}
    if op == "stokes":
        v, psi, sigma, _ = il.solve_stokes(s.cache, s.plus, s.minus, tol=1e-11, maxiter=20000)
        return {"v": v.data, "psi": psi.data, "sigma": sigma.data}
    if s.case["setup"]:
        f, x = _batch_solver(s).solve(s.fp, s.fm, tol=BATCH_TOL)
    else:
        f, x = s.solver.solve(s.fp, s.fm, s.f, s.s, tol=BATCH_TOL)
    return {"f": f, "s": x}


# ---------------------------------------------------------------------------------------------------------------
# the least work of one pass
# ---------------------------------------------------------------------------------------------------------------
def _fft_flops(nx, ny):
    """A zero-padded real convolution: a forward and an inverse real 2-D transform of (2 nx) x (2 ny)."""
    p = 4.0 * nx * ny
    return 2 * 2.5 * p * math.log2(p) + p


def work(case):
    op, es = case["op"], 8 if case["dtype"] == "float64" else 4
    if op == "batch":
        problems = [_batch_problem(i) for i in range(case["problems"])]
        n, pts = [p["nx"] for p in problems], [p["pts"] for p in problems]
        fields, conv = sum(m * m for m in n), sum(_fft_flops(m, m) for m in n)
        matrix = sum(p * p for p in pts)
        return {"bytes": 4.0 * fields + 8.0 * matrix + 12.0 * sum(pts), "flops": (2 if case["setup"] else 1) * conv
                + matrix * (2 * 12 + (250 if case["setup"] else 2))}
    nx, ny = case["nx"], case["ny"]
    cells, pts = float(nx * ny), float(case.get("pts", 0))
    conv = _fft_flops(nx, ny)
    if op == "layer":
        return {"bytes": es * (2 * cells + 2 * pts), "flops": conv + 3 * cells + 64 * pts}
    if op == "calculus":
        return {"bytes": es * cells * (4 + 11), "flops": cells * (2 + 3 + 2 + 3 + 6 + 24 + 10)}
    if op == "invlap":
        return {"bytes": es * 2 * cells, "flops": conv}
    if op == "helmholtz":
        return {"bytes": es * 4 * cells, "flops": 2 * conv + 6 * cells}
    if op in ("dirichlet", "moving"):
        return {"bytes": es * cells + 8 * pts * pts + es * 3 * pts,
                "flops": 2 * conv + 60 * pts * pts + (170 * pts * pts if op == "moving" else 0)}
    if op == "neumann":
        return {"bytes": es * 2 * cells + 8 * pts * pts + es * 4 * pts, "flops": 3 * conv + 60 * pts * pts}
    if op == "heat":
        return {"bytes": es * 2 * cells * case["steps"], "flops": 150.0 * cells * case["steps"]}
    return {"bytes": es * 3 * cells + es * 6 * pts, "flops": 2 * 20 * conv}


# ---------------------------------------------------------------------------------------------------------------
# FP64 restatement in plain torch
# ---------------------------------------------------------------------------------------------------------------
def _yang3(r):
    """The smoothed 3-point kernel of Yang, Zhang, Li and Yang (2009)."""
    r = r.abs()
    s3, r1, r2 = math.sqrt(3.0), r.clamp(max=1.0), r.clamp(1.0, 2.0)
    near = (17 / 48 + s3 * math.pi / 108 + r1 / 4 - r1 * r1 / 4
            + (1 - 2 * r1) / 16 * torch.sqrt((-12 * r1 * r1 + 12 * r1 + 1).clamp(min=0))
            - s3 / 12 * torch.asin((s3 / 2 * (2 * r1 - 1)).clamp(-1, 1)))
    far = (55 / 48 - s3 * math.pi / 108 - 13 * r2 / 12 + r2 * r2 / 4
           + (2 * r2 - 3) / 48 * torch.sqrt((-12 * r2 * r2 + 36 * r2 - 23).clamp(min=0))
           + s3 / 36 * torch.asin((s3 / 2 * (2 * r2 - 3)).clamp(-1, 1)))
    return torch.where(r <= 1, near, torch.where(r < 2, far, torch.zeros_like(r)))


def _lgf(M):
    """G(m, n), 0 <= m, n <= M, of the 5-point Laplacian from its integral representation (G(0, 0) = 0)."""
    xg, wg = np.polynomial.legendre.leggauss(24)
    edges = np.concatenate([[0.0], math.pi * 2.0 ** -np.arange(40, -1, -1.0)])
    half, mid = 0.5 * np.diff(edges), 0.5 * (edges[1:] + edges[:-1])
    a = torch.as_tensor((half[:, None] * xg + mid[:, None]).ravel(), device="cuda")
    w = torch.as_tensor((half[:, None] * wg).ravel(), device="cuda")
    u = 2 * torch.sin(0.5 * a) ** 2
    sh = torch.sqrt(u * (u + 2))
    s, w = torch.log1p(u + sh), w / sh
    k = torch.arange(M + 1, dtype=torch.float64, device="cuda")
    one = (-torch.expm1(-k[:, None] * s)) @ w
    two = (torch.exp(-k[:, None] * s) * w) @ (2 * torch.sin(0.5 * k[:, None] * a) ** 2).T
    g = torch.tril((one[:, None] + two) / (2 * math.pi))   # row q = max, column p = min
    return g + torch.tril(g, -1).T


class _Plain:
    """Grid, points and operators in FP64; fields are (..., n2, n1), x last."""

    def __init__(self, nx, ny, h, i0, bl=None, table=None):
        self.nx, self.ny, self.h, self.i0, self.spec, self.table = nx, ny, h, i0, {}, table
        if bl is not None:
            self.x, self.y, self.n_x, self.n_y, self.ds = (_dev(a, torch.float64)
                                                           for a in (bl.x, bl.y, bl.nx, bl.ny, bl.ds))

    def shape(self, pc):
        dx, dy = _SHAPES[pc]
        return self.ny - 1 + dy, self.nx - 1 + dx

    def window(self, axis, dual):
        """Base index and the 4 weights of every point along one axis."""
        r = (self.x, self.y)[axis] / self.h + self.i0[axis] - (0.5 if dual else 1.0)
        i = r.floor()[:, None] - 1 + torch.arange(4, device="cuda")
        return i.long(), _yang3(i - r[:, None])

    def taps(self, pc):
        dx, dy = _SHAPES[pc]
        (ix, wx), (iy, wy) = self.window(0, dx), self.window(1, dy)
        flat = (iy[:, :, None] * self.shape(pc)[1] + ix[:, None, :]).reshape(len(ix), 16)
        return flat, (wy[:, :, None] * wx[:, None, :]).reshape(len(ix), 16)

    def reg(self, f, pc):
        flat, w = self.taps(pc)
        v = f * (self.ds / self.h ** 2)
        out = torch.zeros(f.shape[:-1] + (self.shape(pc)[0] * self.shape(pc)[1],), dtype=torch.float64, device="cuda")
        out.index_add_(-1, flat.reshape(-1), (v[..., :, None] * w).reshape(f.shape[:-1] + (-1,)))
        return out.reshape(f.shape[:-1] + self.shape(pc))

    def interp(self, q, pc):
        flat, w = self.taps(pc)
        return (q.reshape(q.shape[:-2] + (-1,))[..., flat] * w).sum(-1)

    def linv(self, w):
        n2, n1 = w.shape[-2:]
        p2, p1 = 2 * n2, 2 * n1
        if (n2, n1) not in self.spec:
            if self.table is None:
                self.table = _lgf(max(self.nx, self.ny) + 2)
            i2, i1 = (torch.minimum(k, len(k) - k) for k in (torch.arange(p2, device="cuda"),
                                                             torch.arange(p1, device="cuda")))
            self.spec[n2, n1] = torch.fft.rfft2(self.table[i2[:, None], i1[None, :]]).real
        out = torch.fft.irfft2(torch.fft.rfft2(w, s=(p2, p1)) * self.spec[n2, n1], s=(p2, p1))
        return out[..., :n2, :n1] * self.h ** 2

    # stencils, with the 1/h of grid scaling
    def div(self, u, v):
        return (u[..., :, 1:] - u[..., :, :-1] + v[..., 1:, :] - v[..., :-1, :]) / self.h

    def grad(self, p):
        pad = torch.nn.functional.pad
        return pad((p[..., :, 1:] - p[..., :, :-1]) / self.h, (1, 1)), pad((p[..., 1:, :] - p[..., :-1, :]) / self.h,
                                                                           (0, 0, 1, 1))

    def curl_d(self, s):
        return (s[..., 1:, :] - s[..., :-1, :]) / self.h, (s[..., :, :-1] - s[..., :, 1:]) / self.h

    def curl_e(self, u, v):
        w = (v[..., 1:-1, 1:] - v[..., 1:-1, :-1] - u[..., 1:, 1:-1] + u[..., :-1, 1:-1]) / self.h
        return torch.nn.functional.pad(w, (1, 1, 1, 1))

    # layer operators of scalar data
    def surf_div(self, f):
        return self.div(self.reg(self.n_x * f, "U"), self.reg(self.n_y * f, "V"))

    def normal(self, u, v):
        return self.n_x * self.interp(u, "U") + self.n_y * self.interp(v, "V")

    def cross(self, u, v):
        return self.n_x * self.interp(v, "V") - self.n_y * self.interp(u, "U")

    def columns(self, n, apply, block=16):
        eye = torch.eye(n, dtype=torch.float64, device="cuda")
        return torch.cat([apply(eye[k:k + block]) for k in range(0, n, block)]).T

    def pair_matrix(self, idx, idy, w):
        """sum_ab w_k[a] G(|idx_k[a] - idx_l[b]|, |idy ...|) w_l[b] ds_l: W S for functionals of short stencils."""
        if self.table is None:
            self.table = _lgf(max(self.nx, self.ny) + 2)
        S = torch.zeros(len(w), len(w), dtype=torch.float64, device="cuda")
        for a in range(w.shape[1]):
            dx = (idx[:, a, None, None] - idx[None]).abs()
            dy = (idy[:, a, None, None] - idy[None]).abs()
            S += w[:, a, None] * (self.table[dy, dx] * w[None]).sum(-1)
        return S * self.ds

    def dirichlet_matrix(self):   # E L^-1 R
        (ix, wx), (iy, wy) = self.window(0, 0), self.window(1, 0)
        return self.pair_matrix(ix.repeat(1, 4), iy.repeat_interleave(4, 1),
                                (wy[:, :, None] * wx[:, None, :]).reshape(-1, 16))

    def neumann_matrix(self):     # -C_s L^-1 C_s^T, by the curl stencil of every window on the dual nodes
        parts = []
        for n, ax, dx, dy, sgn in ((self.n_x, 1, 1, 0, 1.0), (self.n_y, 0, 0, 1, -1.0)):
            (ix, wx), (iy, wy) = self.window(0, dx), self.window(1, dy)
            jx, jy = ix.repeat(1, 4), iy.repeat_interleave(4, 1)
            w = sgn * n[:, None] / self.h * (wy[:, :, None] * wx[:, None, :]).reshape(-1, 16)
            parts += [(jx + (ax == 0), jy + (ax == 1), w), (jx, jy, -w)]
        return -self.pair_matrix(*(torch.cat([p[k] for p in parts], 1) for k in range(3)))

    def dirichlet(self, plus, minus):
        fs = self.linv(self.surf_div(plus - minus))
        x = torch.linalg.solve(self.dirichlet_matrix(), 0.5 * (plus + minus) - self.interp(fs, "P"))
        return fs + self.linv(self.reg(x, "P")), x

    def neumann(self, plus, minus, full=True):
        fs = self.linv(self.reg(plus - minus, "P"))
        S = self.neumann_matrix()
        df = torch.linalg.solve(S, self.normal(*self.grad(fs)) - 0.5 * (plus + minus))
        f = fs + self.linv(self.surf_div(df))
        if not full:
            return f, df
        dpsi = torch.linalg.solve(S, self.cross(*self.grad(fs)))
        rhs = self.curl_e(self.reg(self.n_x * df, "U"), self.reg(self.n_y * df, "V")) \
            - self.curl_e(self.reg(self.n_y * dpsi, "U"), self.reg(-self.n_x * dpsi, "V"))
        return f, df, self.linv(rhs), dpsi


def _plain(case, seed):
    g = _grid(case)
    return _Plain(g.nx, g.ny, g.h, g.i0, _bodies(case, seed) if "pts" in case else None)


def _flat(*parts):
    return torch.cat([p.reshape(-1) for p in parts])


def _rounded(a, case):
    """The values that the program's inputs have after their conversion to its type."""
    return _dev(a, DT[case["dtype"]]).double()


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        return _exact_batch(case, seed)
    P, dt = _plain(case, seed), DT[case["dtype"]]
    field = lambda pc, k: _field(case, seed, pc, k, dt).double().reshape(P.shape(pc))  # noqa: E731
    if op == "invlap":
        return P.linv(field("P", 0)).reshape(-1)
    if op == "calculus":
        return _exact_calculus(P, field)
    bl = _bodies(case, seed)
    if op == "layer":
        theta = P.surf_div(_rounded(_surface(bl, seed)[0], case))
        w = P.linv(theta)
        return {"theta": theta.reshape(-1), "w": w.reshape(-1), "g": P.interp(w, "P")}
    if op == "helmholtz":
        dx, dy = (_rounded(a, case) for a in _surface(bl, seed, 2))
        psi = -P.linv(field("D", 0) + P.reg(P.n_x * dy - P.n_y * dx, "D"))
        phi = P.linv(field("P", 1) + P.reg(P.n_x * dx + P.n_y * dy, "P"))
        (cu, cv), (gu, gv) = P.curl_d(psi), P.grad(phi)
        return _flat(cu + gu + 0.3, cv + gv - 0.2)
    if op in ("dirichlet", "moving", "neumann"):
        plus, minus = (_rounded(a, case) for a in _surface(bl, seed, 2))
        if op == "neumann":
            f, df, psi, dpsi = P.neumann(plus, minus)
            return {"f": f.reshape(-1), "df": df, "psi": psi.reshape(-1), "dpsi": dpsi}
        f, x = P.dirichlet(plus, minus)
        return {"f": f.reshape(-1), "s": x}
    if op == "heat":
        return {"T": _exact_heat(P, case, field("P", 0), *(_dev(a, torch.float64) for a in _surface(bl, seed, 2)))}
    return _exact_stokes(P, *(_rounded(a, case) for a in _velocities(bl, seed)))


def _exact_calculus(P, field):
    p, d = field("P", 0), field("D", 1)
    u, v = field("U", 2), field("V", 3)
    pad = torch.nn.functional.pad
    lap = pad((p[1:-1, 2:] + p[1:-1, :-2] + p[2:, 1:-1] + p[:-2, 1:-1] - 4 * p[1:-1, 1:-1]) / P.h ** 2, (1, 1, 1, 1))
    x2p = lambda a: 0.5 * (a[:, 1:] + a[:, :-1])  # noqa: E731  dual -> primal along x, and so on
    y2p = lambda a: 0.5 * (a[1:] + a[:-1])  # noqa: E731
    x2d = lambda a: pad(x2p(a), (1, 1))  # noqa: E731
    y2d = lambda a: pad(y2p(a), (0, 0, 1, 1))  # noqa: E731
    dudx, dvdy = (u[:, 1:] - u[:, :-1]) / P.h, (v[1:] - v[:-1]) / P.h
    dudy = pad((u[1:, 1:-1] - u[:-1, 1:-1]) / P.h, (1, 1, 1, 1))
    dvdx = pad((v[1:-1, 1:] - v[1:-1, :-1]) / P.h, (1, 1, 1, 1))
    cu = x2d(x2p(u) * dudx) + y2p(x2d(v) * dudy)
    cv = x2p(y2d(u) * dvdx) + y2d(y2p(v) * dvdy)
    cu[:, 0] = cu[:, -1] = 0
    cv[0] = cv[-1] = 0
    return [_flat(*P.grad(p)), P.div(u, v).reshape(-1), _flat(*P.curl_d(d)), P.curl_e(u, v).reshape(-1),
            lap.reshape(-1), _flat(cu, cv), _flat(y2p(-x2d(v) * d), x2p(y2d(u) * d))]


def _exact_heat(P, case, T, tp, tm):
    """IF-HERK (Liska and Colonius, scheme A) with dense integrating factors and stage systems."""
    dt, h = 0.5 * P.h ** 2, P.h
    n2, n1 = T.shape

    def kernel(n, a):   # e^{-2a} I_m(2a) as a Toeplitz matrix, by the Fourier integral of the lattice heat kernel
        th = 2 * math.pi * torch.arange(256, dtype=torch.float64, device="cuda") / 256
        m = torch.arange(64, dtype=torch.float64, device="cuda")
        k = (torch.cos(m[:, None] * th) * torch.exp(-2 * a * (1 - torch.cos(th)))).mean(1)
        d = (torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")).abs()
        t = k[d.clamp(max=63)]
        return t * ((d < 64) & (t > 1e-18))

    K = {t: (kernel(n1, 0.5 * t), kernel(n2, 0.5 * t)) for t in (1 / 3, 2 / 3, 1.0)}
    IF = lambda w, t: K[t][1] @ w @ K[t][0]  # noqa: E731

    def dense(axis, n):
        i, w = P.window(axis, 0)
        return torch.zeros(len(i), n, dtype=torch.float64, device="cuda").scatter_(1, i, w)

    Wx, Wy = dense(0, n1), dense(1, n2)
    S = {t: ((Wx @ K[t][0]) @ Wx.T) * ((Wy @ K[t][1]) @ Wy.T) * (P.ds / h ** 2) for t in (1 / 3, 2 / 3)}
    S[0] = (Wx @ Wx.T) * (Wy @ Wy.T) * (P.ds / h ** 2)
    E, R = (lambda q: P.interp(q, "P")), (lambda s: P.reg(s, "P"))
    avg, r1 = 0.5 * (tp + tm), -P.surf_div(tp - tm)
    solve = torch.linalg.solve
    for _ in range(case["steps"]):
        y = IF(T + dt / 3 * r1, 1 / 3)
        s1 = solve(S[1 / 3], (avg - E(y)) / (dt / 3))
        y = IF(IF(T - dt * (r1 + R(s1)), 1 / 3) + 2 * dt * r1, 2 / 3)
        s2 = solve(S[2 / 3], (avg - E(y)) / (2 * dt))
        y = IF(T, 1.0) + IF(0.75 * dt * (r1 + R(s2)), 2 / 3) + 0.25 * dt * r1
        T = y + 0.25 * dt * R(solve(S[0], (avg - E(y)) / (0.25 * dt)))
    return T.reshape(-1)


def _exact_stokes(P, plus, minus):
    """The block-LU Stokes solve with dense Schur complements, column by column."""
    n = len(P.ds)
    dv, vb = plus - minus, 0.5 * (plus + minus)
    dx, dy = dv[:n], dv[n:]
    # symmetric double layer: the tensor n v + v n - (n . v) I on the velocity gradient's positions
    pad, h = torch.nn.functional.pad, P.h
    t11, t12 = P.reg(P.n_x * dx - P.n_y * dy, "P"), P.reg(P.n_y * dx + P.n_x * dy, "D")
    t22 = P.reg(P.n_y * dy - P.n_x * dx, "P")
    fu = pad((t11[:, 1:] - t11[:, :-1] + t12[1:, 1:-1] - t12[:-1, 1:-1]) / h, (1, 1))
    fv = pad((t12[1:-1, 1:] - t12[1:-1, :-1] + t22[1:] - t22[:-1]) / h, (0, 0, 1, 1))
    psi_s = -P.linv(P.linv(P.curl_e(fu, fv)))
    phi = P.linv(P.reg(P.n_x * dx + P.n_y * dy, "P"))
    gu, gv = P.grad(phi)
    E = lambda u, v: torch.cat([P.interp(u, "U"), P.interp(v, "V")], -1)  # noqa: E731
    Ct = lambda s: P.curl_e(P.reg(s[..., :n], "U"), P.reg(s[..., n:], "V"))  # noqa: E731
    S = -P.columns(2 * n, lambda e: E(*P.curl_d(P.linv(P.linv(Ct(e))))))
    sigma = torch.linalg.solve(S, vb - E(gu, gv) - E(*P.curl_d(psi_s)))
    psi = psi_s - P.linv(P.linv(Ct(sigma)))
    cu, cv = P.curl_d(psi)
    d = torch.linalg.solve(P.neumann_matrix(), P.cross(gu, gv))
    psi = psi - P.linv(P.curl_e(P.reg(P.n_y * d, "U"), P.reg(-P.n_x * d, "V")))
    for _ in range(2):   # filter: E R with its rows scaled to sum to one
        parts = []
        for pc, s in (("U", sigma[:n]), ("V", sigma[n:])):
            parts.append(P.interp(P.reg(s, pc), pc) / P.interp(P.reg(torch.ones_like(s), pc), pc))
        sigma = torch.cat(parts)
    return {"v": _flat(cu + gu, cv + gv), "psi": psi.reshape(-1), "sigma": sigma}


def _exact_batch(case, seed):
    table, fields, strengths = _lgf(max(BATCH_SIZES) + 2), [], []
    for p in _batch_specs(case, seed):
        P = _Plain(p.nx, p.ny, p.h, p.i0, p.bl, table)
        plus = _rounded(p.fplus, case)
        f, x = (P.dirichlet(plus, 0 * plus) if p.kind == DIRICHLET else P.neumann(plus, 0 * plus, full=False))
        fields.append(f.reshape(-1))
        strengths.append(x)
    return {"f": torch.cat(fields), "s": torch.cat(strengths)}
