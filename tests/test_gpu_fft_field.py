"""FP32 inverse Laplacian of one field against a zero-padded FP64 FFT
convolution in plain torch.

Tolerance: FP32 transforms forth and back over both directions, 4 log2(8192)
= 52 roundings of eps = 6e-8 relative to the field's 2-norm: 3.1e-6, and as
much again for the spectrum and the split of the real transforms."""
import pytest
import torch

import immersedlayers as il
from test_gpu_sine import _reference

pytestmark = pytest.mark.gpu


# padded sizes from 64 to 8192 x 6144, full and nearly empty padding, odd sizes: the
# general kernels, and from 2048 on both sides those of single fields, all of which
# the next test reaches
@pytest.mark.parametrize("nx,ny", [(30, 70), (65, 34), (70, 40), (100, 65), (110, 97), (140, 130), (1025, 1024), (900, 1025), (1400, 1400), (2000, 1200), (2900, 600), (200, 1100),
                                   (4096, 800), (300, 1500), (600, 800), (500, 900), (1500, 140), (1500, 100),
                                   (1500, 300), (1500, 250), (1500, 500), (250, 2050), (260, 3000), (250, 3072)])
def test_inverse_laplacian_f32(cuda, nx, ny):
    grid = il.PhysicalGrid.from_cells(nx, 0.5, ny=ny)
    c = il.SurfaceScalarCache(None, grid, dtype=torch.float32)
    g = torch.Generator(device="cuda").manual_seed(nx * 10000 + ny)
    f = torch.randn(ny - 1, nx - 1, dtype=torch.float32, device=cuda, generator=g) + 0.3
    w = il.NodesPrimal(grid, f.reshape(-1).clone())
    out = il.NodesPrimal.zeros(grid, torch.float32)
    il.inverse_laplacian_(out, w, c)
    ref = _reference(f.double()) * 0.25   # 1 / factor = h^2
    err = float((out.component(0).double() - ref).norm() / ref.norm())
    assert err <= 6e-6, err
    il.inverse_laplacian_(w, c)  # in place
    assert torch.equal(w.data, out.data)


# every row length (1024, 1536, .. 4096) and column length (2048, 3072, 4096, 6144) of
# the single-field kernels, at the fewest and the most values that take it, odd sizes
@pytest.mark.parametrize("nx,ny", [(770, 770), (1025, 1025), (1026, 900), (1537, 1026), (1538, 800), (2049, 1537),
                                   (2050, 770), (3073, 900), (3074, 1026), (900, 1538), (1025, 2049), (1030, 2050),
                                   (1100, 3073), (4097, 3073)])
def test_inverse_laplacian_f32_instances(cuda, nx, ny):
    test_inverse_laplacian_f32(cuda, nx, ny)
