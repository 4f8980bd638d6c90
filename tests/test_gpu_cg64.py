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
# the inverse, either side of the cluster / grid rule (256 unknowns), a partial
# last slice, a slice too large for shared memory; points 0.45 h apart (S
# numerically singular: the inverse is refused or useless, and the CG runs)
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
