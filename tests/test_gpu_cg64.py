"""FP64 CG of one dense Schur complement: sizes around its slices and variants.

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


# fewer points than CTAs, one row per CTA, either side of the cluster / grid
# rule (256 unknowns), a partial last slice, a slice too large for shared memory
@pytest.mark.parametrize("n", [3, 16, 131, 256, 257, 700, 1870])
def test_dense_cg_residual(cuda, n):
    grid = il.PhysicalGrid.from_cells(max(64, int(n / 1.79)), 4.0 / max(64, int(n / 1.79)))
    bl = il.BodyList().append(il.circle(min(1.6, n * 1.4 * grid.h / (2 * np.pi)), n=n))
    c = il.SurfaceScalarCache(bl, grid)
    f = W.fourier_surface_data(bl, np.random.default_rng(n))
    plus = il.ScalarData(torch.tensor(f, device=cuda))
    minus = il.ScalarData(torch.zeros(n, dtype=torch.float64, device=cuda))
    _, s, info = il.solve_dirichlet(c, plus, minus, tol=TOL, maxiter=20000)
    assert info["converged"] and info["rel_residual"] <= TOL
    fs, g = il.zeros_grid(c), il.zeros_surface(c)
    il.surface_divergence_(fs, plus, c)
    il.inverse_laplacian_(fs, c)
    il.interpolate_(g, fs, c)
    b = g.data - 0.5 * plus.data
    r = b - il.create_RTLinvR(c) @ s.data
    assert float(r.norm()) <= (TOL + 1e-12) * float(b.norm())
