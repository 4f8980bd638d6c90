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


@pytest.mark.parametrize("precond", ["none", "bjacobi"])
@pytest.mark.parametrize("variant", [1, 3, 6])
def test_batched_cg_cluster_sizes(cuda, precond, variant):
    """Problems of each queue of the size split (clusters of 16, 8 and 4 CTAs;
    row counts that do not divide), with the coarse correction of several
    bodies: the FP64 residual of every solution meets the tolerance.  The
    kernel's own true residual is formed in float-float, 2^-44 per operation on
    |S| |x|: 1e-10 of |b| beside the 1e-9 asked for."""
    import torch
    import immersedlayers as il
    from immersedlayers import bodies as B
    from immersedlayers.batch import BatchProblemSpec, BatchSolver
    h = 4.0 / 512
    specs = []
    for i, (nb, nper) in enumerate([(1, 5), (1, 33), (3, 47), (2, 97), (1, 193), (3, 129), (2, 201), (1, 401)]):
        for kind in (0, 1):
            bl = B.BodyList()
            for q in range(nb):
                b = B.circle(nper * 1.4 * h / (2 * np.pi), n=nper)
                bl.append(B.Body(b.x + 1.1 * (q - 0.5 * (nb - 1)), b.y + 0.2 * q, b.nx, b.ny, b.ds))
            specs.append(BatchProblemSpec(512, h, bl, kind, np.zeros(len(bl))))
    bs = BatchSolver(specs, dtype=torch.float32)
    if precond == "bjacobi":
        bs.set_precond("bjacobi", 64)
        bs.set_coarse(True)
    bs.set_cg_variant(variant)
    rng = np.random.default_rng(3)
    rhs = torch.tensor(rng.standard_normal(bs.total_points), dtype=torch.float64, device="cuda")
    # smooth data: S times a vector
    rhs = bs.schur_apply(rhs)
    x = bs.schur_solve(rhs, tol=1e-9, maxiter=20000)
    r = bs.schur_apply(x) - rhs
    torch.cuda.synchronize()
    its, rr = bs.info()
    assert (rr <= 1e-9).all(), (its, rr)
    o = bs.point_offsets
    for i in range(len(specs)):
        a, b = o[i], o[i + 1]
        assert r[a:b].norm().item() <= 1.1e-9 * rhs[a:b].norm().item(), (i, its[i])


def test_batched_solve_queues(cuda):
    """A batch whose default solve runs in three queues (16, 8 and 4 CTAs per
    problem) against the same batch on clusters of 8: both to a residual of
    1e-10, so the fields agree to 1e-8 (the strengths of the slow modes, up to a
    condition number of 1e5 off, act on the field by their small eigenvalues)."""
    import torch
    from immersedlayers import bodies as B
    from immersedlayers.batch import BatchProblemSpec, BatchSolver
    h = 4.0 / 512
    rng = np.random.default_rng(8)
    specs = []
    for n in (9, 150, 193, 260, 385, 410):
        for kind in (0, 1):
            b = B.circle(n * 1.4 * h / (2 * np.pi), n=n)
            t = 2 * np.pi * np.arange(n) / n
            a = rng.standard_normal(4)
            specs.append(BatchProblemSpec(512, h, b, kind, a[0] * np.cos(t) + a[1] * np.sin(2 * t) + a[2] * np.cos(3 * t)))
    bs = BatchSolver(specs, dtype=torch.float64)
    bs.set_precond("bjacobi", 64)
    bs.set_coarse(True)
    fp, fm = bs.surface_data()
    out = {}
    for variant in (6, 1):
        bs.set_cg_variant(variant)
        f, _ = bs.solve(fp, fm, tol=1e-10, maxiter=20000)
        torch.cuda.synchronize()
        its, rr = bs.info()
        assert (rr <= 1e-10).all(), (variant, its, rr)
        out[variant] = f.clone()
    for i in range(len(specs)):
        a, b = bs.field(out[6], i), bs.field(out[1], i)
        assert (a - b).abs().max().item() <= 1e-8 * b.abs().max().item(), i
