"""Solves where the device grants less than they ask for: CUDA runtime calls of
libilm.so refused by a preloaded library, in a process of their own."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# passes every call on but those it is told to refuse (refuse_*, most_ctas), and counts
# the live device allocations of watch_bytes
SHIM = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stddef.h>
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), name); }
size_t refuse_bytes = 0, watch_bytes = 0;
int refuse_cluster = 0, refuse_attribute = 0, most_ctas = 1 << 30, refused = 0, live = 0;
static void* ptrs[64];
cudaError_t cudaMalloc(void** p, size_t n) {
  if (refuse_bytes && n == refuse_bytes) {
    ++refused;
    /* the runtime's own refusal, so that its last error is set as in earnest */
    return ((cudaError_t (*)(void**, size_t))real("cudaMalloc"))(p, (size_t)1 << 50);
  }
  cudaError_t e = ((cudaError_t (*)(void**, size_t))real("cudaMalloc"))(p, n);
  if (e == 0 && watch_bytes && n == watch_bytes)
    for (int k = 0; k < 64; ++k)
      if (!ptrs[k]) { ptrs[k] = *p; ++live; break; }
  return e;
}
cudaError_t cudaFree(void* p) {
  for (int k = 0; p && k < 64; ++k)
    if (ptrs[k] == p) { ptrs[k] = 0; --live; }
  return ((cudaError_t (*)(void*))real("cudaFree"))(p);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  for (unsigned k = 0; refuse_cluster && k < c->numAttrs; ++k)
    if (c->attrs[k].id == cudaLaunchAttributeClusterDimension && (int)c->attrs[k].val.clusterDim.x >= refuse_cluster) {
      ++refused;
      return cudaErrorInvalidClusterSize;
    }
  return ((cudaError_t (*)(const cudaLaunchConfig_t*, const void*, void**))real("cudaLaunchKernelExC"))(c, f, args);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  if (refuse_cluster && a == cudaFuncAttributeNonPortableClusterSizeAllowed && refuse_attribute) {
    ++refused;
    return cudaErrorNotSupported;
  }
  return ((cudaError_t (*)(const void*, enum cudaFuncAttribute, int))real("cudaFuncSetAttribute"))(f, a, v);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, struct dim3 g, struct dim3 b, void** args, size_t sm, cudaStream_t st) {
  if ((int)g.x > most_ctas) {
    ++refused;
    return cudaErrorCooperativeLaunchTooLarge;
  }
  return ((cudaError_t (*)(const void*, struct dim3, struct dim3, void**, size_t, cudaStream_t))real(
      "cudaLaunchCooperativeKernel"))(f, g, b, args, sm, st);
}
"""

HEAD = r"""
import ctypes as C, os, sys
sys.path[:0] = [os.path.join(ROOT, p) for p in ("immersedlayers.jl_gb300", "oracle", "tests")]
import numpy as np, torch
import immersedlayers as il
from immersedlayers import workloads as W
shim = C.CDLL(SHIM)

def setting(name, typ=C.c_size_t):
    return typ.in_dll(shim, name)

def inverse_bytes(n):
    nt = (n + 31) // 32
    return nt * 32 * (nt * 32 + 32) * 4

def case(n):
    nx = max(64, int(n / 1.79))
    grid = il.PhysicalGrid.from_cells(nx, 4.0 / nx)
    bl = il.BodyList().append(il.circle(min(1.6, n * 1.4 * grid.h / (2 * np.pi)), n=n))
    c = il.SurfaceScalarCache(bl, grid)
    f = W.fourier_surface_data(bl, np.random.default_rng(n))
    return grid, bl, c, il.ScalarData(torch.tensor(f, device="cuda")), il.ScalarData(torch.zeros(n, dtype=torch.float64, device="cuda"))

def true_residual(c, plus, s):
    fs, g = il.zeros_grid(c), il.zeros_surface(c)
    il.surface_divergence_(fs, plus, c)
    il.inverse_laplacian_(fs, c)
    il.interpolate_(g, fs, c)
    b = g.data - 0.5 * plus.data
    return float((b - il.create_RTLinvR(c) @ s.data).norm() / b.norm())

def heat(grid, bl):
    one = lambda t, x, c, p, m: il.ones_surface(c)
    prob = il.DirichletHeatConductionProblem(grid, bl, dtype=torch.float64, phys_params={"diffusivity": 1.0, "Fourier": 0.5},
                                             bc={"exterior": one, "interior": one}, timestep_func=il.timestep_fourier)
    system = il.construct_system(prob)
    return il.init(il.init_sol(system), (0.0, 1.0), system, tol=1e-11, maxiter=2000)
"""


@pytest.fixture(scope="module")
def child(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    src, shim = str(d / "shim.c"), str(d / "shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    from immersedlayers import _build
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    subprocess.run(["gcc", "-shared", "-fPIC", "-I" + inc, "-o", shim, src, "-ldl"], check=True, capture_output=True)

    def run(body):
        code = f"ROOT, SHIM = {ROOT!r}, {shim!r}\n" + HEAD + textwrap.dedent(body)
        r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=shim), capture_output=True,
                           text=True, timeout=240)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return run


@pytest.mark.parametrize("n", [150, 300])
def test_solve_without_memory_for_the_inverse(child, n):
    """No memory for the FP32 inverse: the FP64 CG alone solves (n on either side
    of its cluster / grid rule), single solves and a heat march."""
    child(f"""
    n = {n}
    grid, bl, c, plus, minus = case(n)
    setting("refuse_bytes").value = inverse_bytes(n)
    _, s, info = il.solve_dirichlet(c, plus, minus, tol=1e-10, maxiter=20000)
    assert setting("refused", C.c_int).value == 1
    assert info["converged"] and true_residual(c, plus, s) <= 1e-10 + 1e-12
    integ = heat(grid, bl)
    integ.advance(2)
    assert setting("refused", C.c_int).value == 4
    assert max(integ.info()["rel_residual"]) <= 1e-11 and max(integ.info()["iterations"]) > 5
    setting("refuse_bytes").value = 0
    full = heat(grid, bl)
    full.advance(2)
    a, b = integ.u.state.data, full.u.state.data
    # two solves of 1e-11 per stage, condition of the stage systems below 10 at 1.4 h
    assert float((a - b).abs().max()) <= 1e-9 * float(b.abs().max())
    """)


def test_memory_of_the_inverses(child):
    """One matrix per system and one to form them in: two Poisson systems of a
    cache keep three, a heat march keeps its three inverses."""
    child("""
    n = 150
    grid, bl, c, plus, minus = case(n)
    setting("watch_bytes").value = inverse_bytes(n)
    live = setting("live", C.c_int)
    il.solve_dirichlet(c, plus, minus)
    il.solve_neumann(c, plus, minus)
    assert live.value == 3, live.value
    integ = heat(grid, bl)
    integ.advance(1)
    assert live.value == 6, live.value
    """)


@pytest.mark.parametrize("n,most,refusals", [(150, 152, 1), (256, 4, 6), (400, 9, 4), (700, 8, 5), (700, 100, 1)])
def test_solve_on_fewer_sms(child, n, most, refusals):
    """No cluster of 16 and at most `most` CTAs of a cooperative launch: the solve
    takes the grid, and half as many CTAs until they fit (S in shared memory, or
    with 700 points on 4 CTAs streamed from L2)."""
    child(f"""
    n = {n}
    grid, bl, c, plus, minus = case(n)
    setting("refuse_cluster", C.c_int).value = 16
    setting("most_ctas", C.c_int).value = {most}
    _, s, info = il.solve_dirichlet(c, plus, minus, tol=1e-10, maxiter=20000)
    assert setting("refused", C.c_int).value == {refusals}, setting("refused", C.c_int).value
    assert info["converged"] and true_residual(c, plus, s) <= 1e-10 + 1e-12
    integ = heat(grid, bl)
    integ.advance(2)
    assert max(integ.info()["rel_residual"]) <= 1e-11
    """)


def test_batch_without_large_clusters(child):
    """A batch whose largest problem would take a cluster of 16 CTAs takes one of 8."""
    child("""
    from immersedlayers.batch import BatchProblemSpec, BatchSolver
    n = 400
    grid, bl, c, plus, minus = case(n)
    sol = []
    for refuse in (0, 16):
        setting("refuse_cluster", C.c_int).value = setting("refuse_attribute", C.c_int).value = refuse
        bs = BatchSolver([BatchProblemSpec(grid.nx, grid.h, bl, 0, plus.data.cpu().numpy())], dtype=torch.float64)
        _, s = bs.solve(*bs.surface_data(), tol=1e-9, maxiter=5000)
        assert (bs.info()[1] <= 1e-9).all()
        sol.append(s.clone())
    assert setting("refused", C.c_int).value > 0
    # two solutions of relative residual 1e-9, condition some 1e3
    assert float((sol[0] - sol[1]).norm()) <= 1e-5 * float(sol[0].norm())
    """)
