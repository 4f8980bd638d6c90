"""The device set-up kernels at their edges: tile lists of every length class
after a re-binning, and the batched pair sums with and without the LGF patch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts", [1, 7, 33, 128, 129, 700])
def test_rebinned_tile_lists(cuda, npts):
    """Points crowded into a few tiles (lists of 1 to 700 points), given in
    random order: the scatter of a re-binned cache sums every cell's points in
    the order of a cache built there by the host, so the fields are equal."""
    import torch
    import immersedlayers as il
    from immersedlayers import bodies as B
    g = il.PhysicalGrid((-1.0, 1.0), (-1.0, 1.0), 0.02)
    rng = np.random.default_rng(npts)

    def points(x0, r):
        t = 2 * np.pi * rng.permutation(npts) / npts
        return (x0 + r * np.cos(t), 0.1 + r * np.sin(t), np.cos(t), np.sin(t), np.full(npts, 0.01))
    moving = il.SurfaceScalarCache(B.Body(*points(-0.4, 0.3)), g, dtype=torch.float64)
    new = points(0.35, 0.05)
    moving.update_points_(*new)
    fresh = il.SurfaceScalarCache(B.Body(*new), g, dtype=torch.float64)
    f = il.ScalarData(torch.tensor(rng.standard_normal(npts), dtype=torch.float64, device="cuda"))
    for make, op in [(il.zeros_grid, il.regularize_), (il.zeros_grid, il.surface_divergence_)]:
        a, b = op(make(moving), f, moving).data, op(make(fresh), f, fresh).data
        torch.cuda.synchronize()
        # windows from the same formulas, device against host math functions: 1e-13
        assert (a - b).abs().max().item() <= 1e-13 * b.abs().max().item()


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("sep,nper", [(0.0, 31), (1.5, 24), (0.2, 8)])
def test_batched_pair_sums_match_dense(cuda, kind, sep, nper):
    """S x of a batch problem (float-float pair sums) against the dense FP64
    Schur complement: one body (every tile's distances fit the patch), bodies
    far apart (tiles across bodies read the table), a partial last tile.
    Some 500 float-float operations of 2^-44 on differences of weights: 1e-11
    of |S| |x|."""
    import torch
    import immersedlayers as il
    from immersedlayers import bodies as B
    from immersedlayers.batch import BatchProblemSpec, BatchSolver
    h, nx = 4.0 / 256, 256
    bl = B.BodyList()
    r = nper * 1.4 * h / (2 * np.pi)
    for s in ([0.0] if sep == 0.0 else [-sep, sep]):
        b = B.circle(r, n=nper)
        bl.append(B.Body(b.x + s, b.y + 0.3 * s, b.nx, b.ny, b.ds))
    n = len(bl)
    bs = BatchSolver([BatchProblemSpec(nx, h, bl, kind, np.zeros(n))], dtype=torch.float64)
    g = il.PhysicalGrid(h=h, nx=nx)
    x = torch.tensor(np.random.default_rng(n).standard_normal(n), dtype=torch.float64, device="cuda")
    y = bs.schur_apply(x)
    c = il.SurfaceScalarCache(bl, g, dtype=torch.float64)
    S = (il.create_RTLinvR if kind == 0 else il.create_CLinvCT)(c)
    torch.cuda.synchronize()
    assert (y - S @ x).abs().max().item() <= 1e-11 * (S.abs() @ x.abs()).max().item()
