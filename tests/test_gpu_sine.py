"""FP64 inverse Laplacian by sine transforms against a zero-padded FFT
convolution with the lattice Green's function in plain FP64 torch.

Tolerance: both sides are transforms with errors of a few eps log2(N) (eps =
1.1e-16, log2 N <= 12) relative to the field's 2-norm; 2e-14 leaves a factor of
four over 3 * 12 * eps."""
import math

import numpy as np
import pytest
import torch

import immersedlayers as il

pytestmark = pytest.mark.gpu


def _lgf(M):
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
    g = torch.tril((one[:, None] + two) / (2 * math.pi))
    return g + torch.tril(g, -1).T


def _reference(f):
    n2, n1 = f.shape
    G = _lgf(max(n1, n2) + 1)
    i2, i1 = (torch.minimum(k, len(k) - k) for k in (torch.arange(2 * n2, device="cuda"),
                                                     torch.arange(2 * n1, device="cuda")))
    S = torch.fft.rfft2(G[i2[:, None], i1[None, :]]).real
    return torch.fft.irfft2(torch.fft.rfft2(f, s=(2 * n2, 2 * n1)) * S, s=(2 * n2, 2 * n1))[:n2, :n1]


# smallest grids; N = n1 + 1 exactly a transform size, one below and above; odd
# row counts; rows at a multiple of the chunk count (64) and either side; both
# stage kinds (N <= 256 and above), both radix-3 sizes; more rows than 64 chunks
# of 32 (the two-mode variant); a box too wide for its height (FFT path)
@pytest.mark.parametrize("nx,ny", [(4, 5), (5, 9), (13, 12), (48, 65), (49, 66), (64, 64), (65, 130), (129, 200),
                                   (192, 193), (193, 257), (256, 129), (257, 300), (300, 450), (385, 320),
                                   (513, 400), (769, 700), (260, 2049), (270, 2060), (900, 60)])
def test_inverse_laplacian_f64(cuda, nx, ny):
    grid = il.PhysicalGrid.from_cells(nx, 0.5, ny=ny)
    c = il.SurfaceScalarCache(None, grid)
    g = torch.Generator(device="cuda").manual_seed(nx * 10000 + ny)
    f = torch.randn(ny - 1, nx - 1, dtype=torch.float64, device=cuda, generator=g) + 0.3
    w = il.NodesPrimal(grid, f.reshape(-1).clone())
    out = il.NodesPrimal.zeros(grid)
    il.inverse_laplacian_(out, w, c)
    ref = _reference(f) * 0.25   # 1 / factor = h^2
    err = float((out.component(0) - ref).norm() / ref.norm())
    assert err <= 2e-14, err
    il.inverse_laplacian_(w, c)  # in place
    assert torch.equal(w.data, out.data)


@pytest.mark.parametrize("nx,ny,rows", [(97, 120, [0]), (97, 120, [118]), (130, 201, [7, 64, 65, 199]), (600, 311, [1]),
                                        (1100, 350, [20, 348]), (49, 66, [])])
def test_inverse_laplacian_rows_of_zeros(cuda, nx, ny, rows):
    """A field that is zero but for some rows (first, last, unpaired ones; none:
    zero out): the pairs of zero rows are not transformed."""
    grid = il.PhysicalGrid.from_cells(nx, 0.5, ny=ny)
    c = il.SurfaceScalarCache(None, grid)
    g = torch.Generator(device="cuda").manual_seed(nx)
    f = torch.zeros(ny - 1, nx - 1, dtype=torch.float64, device=cuda)
    for r in rows:
        f[r] = torch.randn(nx - 1, dtype=torch.float64, device=cuda, generator=g) + 0.3
    out = il.NodesPrimal.zeros(grid)
    out.data.fill_(7.0)
    il.inverse_laplacian_(out, il.NodesPrimal(grid, f.reshape(-1).clone()), c)
    ref = _reference(f) * 0.25
    assert float((out.component(0) - ref).norm()) <= 2e-14 * float(ref.norm())


def test_tables_are_given_back(cuda):
    """Grids of forty heights, one after the other, and the first ones again:
    what stays on the device is bounded (a copy of the lattice Green's function
    per height is 8 MB here, 320 MB in all), and the results are the same.  Tables
    of 64 MB may stay; 32 MB more leaves room for the allocator."""
    def field(ny):
        grid = il.PhysicalGrid.from_cells(64, 0.5, ny=ny)
        c = il.SurfaceScalarCache(None, grid)
        g = torch.Generator(device="cuda").manual_seed(ny)
        w = il.NodesPrimal(grid, torch.randn(63 * (ny - 1), dtype=torch.float64, device=cuda, generator=g))
        return il.inverse_laplacian_(il.NodesPrimal.zeros(grid), w, c).data.clone()
    first = [field(ny) for ny in (1040, 1000)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    for ny in range(1001, 1040):
        field(ny)
    again = [field(ny) for ny in (1040, 1000)]
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(first, again))
    torch.cuda.empty_cache()
    assert free - torch.cuda.mem_get_info()[0] <= 96 << 20
