"""FP64 solve of one dense Schur complement (refined FP32 inverse, then CG):
sizes around its slices, tiles and variants.

The residual is formed from the dense Schur complement of create_RTLinvR by
FP64 torch products; the solve promises ||b - S s|| <= tol ||b||, and the
check's own rounding is below 1e-12 ||b|| (n eps ||S|| ||s|| / ||b||)."""
import pytest
import torch

import immersedlayers as il
from immersedlayers import workloads as W

import numpy as np

pytestmark = pytest.mark.gpu
TOL = 1e-10


# fewer points than CTAs, one row per CTA, whole and partial 32 x 32 tiles of
# the inverse, either side of 256 (the cluster / grid rule of the CG without an
# inverse; the one with it is tested below), a partial last slice, a slice too
# large for shared memory; points 0.45 h apart (S numerically singular: the
# inverse is refused or useless, and the CG runs)
@pytest.mark.parametrize("n,ds", [(3, 1.4), (16, 1.4), (32, 1.4), (33, 1.4), (131, 1.4), (256, 1.4), (257, 1.4),
                                  (700, 1.4), (1870, 1.4), (180, 0.45)])
def test_dense_solve_residual(cuda, n, ds):
    nx = max(64, int(n / 1.79))
    grid = il.PhysicalGrid.from_cells(nx, 4.0 / nx)
    bl = il.BodyList().append(il.circle(min(1.6, n * ds * grid.h / (2 * np.pi)), n=n))
    c = il.SurfaceScalarCache(bl, grid)
    f = W.fourier_surface_data(bl, np.random.default_rng(n))
    plus = il.ScalarData(torch.tensor(f, device=cuda))
    minus = il.ScalarData(torch.zeros(n, dtype=torch.float64, device=cuda))
    tol = TOL if ds > 1 else 1e-4
    _, s, info = il.solve_dirichlet(c, plus, minus, tol=tol, maxiter=20000)
    assert info["converged"] and info["rel_residual"] <= tol
    fs, g = il.zeros_grid(c), il.zeros_surface(c)
    il.surface_divergence_(fs, plus, c)
    il.inverse_laplacian_(fs, c)
    il.interpolate_(g, fs, c)
    b = g.data - 0.5 * plus.data
    r = b - il.create_RTLinvR(c) @ s.data
    assert float(r.norm()) <= (tol + 1e-12) * float(b.norm())


@pytest.mark.parametrize("n,tol", [(131, 1e-1), (131, 1e-4), (700, 1e-4)])
def test_reported_residual_dense(cuda, n, tol):
    """rel_residual is that of the strengths returned (the solver corrects them
    once more after the residual that passes): both variants of the exchange.
    The check's own rounding as above; a norm of rounded differences: 1e-3."""
    nx = max(64, int(n / 1.79))
    grid = il.PhysicalGrid.from_cells(nx, 4.0 / nx)
    bl = il.BodyList().append(il.circle(min(1.6, n * 1.4 * grid.h / (2 * np.pi)), n=n))
    c = il.SurfaceScalarCache(bl, grid)
    f = W.fourier_surface_data(bl, np.random.default_rng(n))
    plus = il.ScalarData(torch.tensor(f, device=cuda))
    minus = il.ScalarData(torch.zeros(n, dtype=torch.float64, device=cuda))
    _, s, info = il.solve_dirichlet(c, plus, minus, tol=tol, maxiter=20000)
    fs, g = il.zeros_grid(c), il.zeros_surface(c)
    il.surface_divergence_(fs, plus, c)
    il.inverse_laplacian_(fs, c)
    il.interpolate_(g, fs, c)
    b = g.data - 0.5 * plus.data
    true = float((b - il.create_RTLinvR(c) @ s.data).norm() / b.norm())
    assert info["converged"] and true <= tol
    assert abs(info["rel_residual"] - true) <= 1e-3 * true + 1e-12


@pytest.mark.parametrize("ds,tol", [(0.58, 0.2), (0.65, 0.2), (0.65, 0.01), (1.0, 1e-4)])
def test_reported_residual_warm_start(cuda, ds, tol):
    """The last stage solve of a heat step that starts from strengths within the
    tolerance (noise of 1e-2 on a slowly changing field; at the smaller
    tolerances, outside it): the constraint E T = 1 misses by dt b3 times the
    residual of the strengths used.  The fields' rounding, 1e-15 / (dt b3), over
    |b| of at least 1e-2 / (dt b3): 1e-10 leaves the rest to S, sums of some 20
    float-float values (2^-48) times strengths of up to 1e3 |b|."""
    from geometry import heat_case
    og, b = heat_case(ds_factor=ds)
    g = il.PhysicalGrid((-1.28, 1.28), (-1.28, 1.28), og.h)
    one = lambda t, x, c, p, m: il.ones_surface(c)
    prob = il.DirichletHeatConductionProblem(g, b, dtype=torch.float64, phys_params={"diffusivity": 1.0, "Fourier": 0.5},
                                             bc={"exterior": one, "interior": one}, timestep_func=il.timestep_fourier)
    system = il.construct_system(prob)
    c = system.base_cache
    integ = il.init(il.init_sol(system), (0.0, 1.0), system, tol=tol, maxiter=2000)
    integ.advance(40)
    T = integ.u.state
    gen = torch.Generator(device="cuda").manual_seed(3)
    T.data.add_(1e-2 * torch.randn(T.data.numel(), generator=gen, device="cuda", dtype=torch.float64))
    integ.advance(1)
    Rs, Ss, ET = il.zeros_grid(c), il.zeros_surface(c), il.zeros_surface(c)
    il.regularize_(Rs, il.ScalarData(-integ.u.constraint.data), c)   # the constraint is -sigma
    il.interpolate_(Ss, Rs, c)
    il.interpolate_(ET, T, c)
    r = (1.0 - ET.data) / (0.25 * integ.dt)
    true = float(r.norm() / (Ss.data + r).norm())
    rep = integ.info()["rel_residual"][2]
    assert true <= tol + 1e-10
    assert abs(rep - true) <= 1e-3 * true + 1e-10, (rep, true)


@pytest.mark.parametrize("n", [320, 321])
def test_dense_solve_either_side_of_the_variants(cuda, n):
    test_dense_solve_residual(cuda, n, 1.4)


@pytest.mark.parametrize("n", [17, 560, 561])
def test_stage_solves_either_side_of_the_variants(cuda, n):
    """The heat march's sparse systems in the cluster and on the grid: every stage
    within its tolerance, and the constraint E T = 1 with it.  The last stage's
    residual is the constraint's over dt b3, its right-hand side the change that a
    step makes there, below 1 / (dt b3): 1e-11, and the fields' rounding."""
    nx = max(64, int(n / 1.79))
    grid = il.PhysicalGrid.from_cells(nx, 4.0 / nx)
    bl = il.BodyList().append(il.circle(min(1.6, n * 1.4 * grid.h / (2 * np.pi)), n=n))
    one = lambda t, x, c, p, m: il.ones_surface(c)
    prob = il.DirichletHeatConductionProblem(grid, bl, dtype=torch.float64,
                                             phys_params={"diffusivity": 1.0, "Fourier": 0.5},
                                             bc={"exterior": one, "interior": one}, timestep_func=il.timestep_fourier)
    system = il.construct_system(prob)
    integ = il.init(il.init_sol(system), (0.0, 1.0), system, tol=1e-11, maxiter=2000)
    for _ in range(3):  # cold, then warm starts
        integ.advance(1)
        assert max(integ.info()["rel_residual"]) <= 1e-11
        ET = il.zeros_surface(system.base_cache)
        il.interpolate_(ET, integ.u.state, system.base_cache)
        assert float((ET.data - 1.0).norm()) <= 1e-11 * n ** 0.5 + 1e-13 * n ** 0.5
