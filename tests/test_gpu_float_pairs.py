"""The integer forms of the FP64 <-> float-float conversions
(ilm_internal.cuh) in a kernel compiled here against exact arithmetic."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "ilm_internal.cuh"
using namespace ilm;
__global__ void k(int n, const double* v, float* hi, float* lo, double* back) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const FF f = split_ff(v[i]);
  hi[i] = f.hi;
  lo[i] = f.lo;
  back[i] = join_ff(f.hi, f.lo);
}
extern "C" __attribute__((visibility("default"))) int run(int n, const double* v, float* hi, float* lo, double* back) {
  k<<<(n + 255) / 256, 256>>>(n, v, hi, lo, back);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(cuda, tmp_path_factory):
    from immersedlayers import _build
    d = tmp_path_factory.mktemp("pairs")
    src, out = str(d / "pairs.cu"), str(d / "pairs.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.FLAGS, "-I" + _build.INCLUDE, "-I" + _build.CSRC, "-shared",
                    src, "-o", out, "-lcudart"], check=True, capture_output=True)
    return C.CDLL(out).run


def test_split_and_join(cuda, run):
    """hi + lo within 2^-49 of v (hi to nearest leaves 28 bits and a sign, of
    which lo keeps 24), and joined without error: all exponents of the integer
    form, carries into the exponent, ties, zeros; the range beyond it is taken by
    conversions (down to FP32's normal numbers times 2^24)."""
    import torch
    rng = np.random.default_rng(7)
    v = rng.standard_normal(1 << 18) * 2.0 ** rng.integers(-72, 126, 1 << 18)
    edge = [m * 2.0 ** e for e in range(-74, 127)
            for m in (1.0, 1 + 2.0 ** -24, 1 + 2.0 ** -23 + 2.0 ** -24, 1 + 2.0 ** -25, 2 - 2.0 ** -52, 2 - 2.0 ** -24,
                      2 - 2.0 ** -25, 1 + 2.0 ** -52, 1.5 - 2.0 ** -30)]
    v = np.concatenate([v, edge, [0.0, -0.0], -np.array(edge)])
    dv = torch.tensor(v, device=cuda)
    hi, lo = (torch.empty(len(v), dtype=torch.float32, device=cuda) for _ in range(2))
    back = torch.empty_like(dv)
    torch.cuda.synchronize()
    assert run(len(v), *(C.c_void_p(t.data_ptr()) for t in (dv, hi, lo, back))) == 0
    h, l = hi.cpu().numpy().astype(np.float64), lo.cpu().numpy().astype(np.float64)
    assert (np.abs((v - h) - l) <= 2.0 ** -49 * np.abs(v)).all()   # both differences are exact
    assert (np.abs(l) <= 2.0 ** -24 * np.abs(h)).all()
    assert (back.cpu().numpy() == h + l).all()
