// Heat conduction with Dirichlet surfaces, marched by IF-HERK on the device.
//
// The reference's DirichletHeatConduction problem (test/literate/
// heatconduction.jl:87-189) is the constrained ODE
//     dT/dt = kappa L T + R sigma - kappa D_s[T],     E T = (T_b+ + T_b-)/2
// advanced by ConstrainedSystems' LiskaIFHERK (src/timemarching.jl:4,262-277):
// an integrating factor exp(tau kappa L) for the Laplacian and a half-explicit
// Runge-Kutta scheme for the constraint, one Schur solve per stage.
//
// Restatement used here (Liska & Colonius IF-HERK, scheme A: c = (0,1/3,1),
// a21 = 1/3, a31 = -1, a32 = 2, b = (0,3/4,1/4)):
//  * exp(a L5) on the unbounded lattice is the separable discrete heat kernel
//    e^{-2a} I_m(2a) per direction (a = kappa tau / h^2), applied as two short
//    1-D stencils (radius <= ~16 for the step sizes used);
//  * every stage needs the constraint only at the surface points, so the
//    stage right-hand sides are point-local gathers (E exp(aL) T is a gather
//    with the DDF window smeared by the heat kernel) and the stage Schur
//    complements S_a = E exp(aL) R are short-range: they are assembled once as
//    sparse matrices (float-float values) and solved with a warm start from
//    the previous step by an FP32 inverse refined with FP64 residuals, FP64 CG
//    where that stalls (ilm_cg64.cu);
//  * the grid is touched once per step: T <- exp(dt kappa L) T +
//    b2 dt exp(2/3 dt kappa L) R sigma_2 + b3 dt R sigma_3 + (constant field).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <new>
#include <unordered_map>

#include "ilm_internal.cuh"

namespace ilm {

namespace {

// e^{-2a} I_m(2a), m = 0..R, by the power series of I_m (a <= ~4)
std::vector<double> heat_kernel_taps(double a, double tol = 1e-17, int rmax = 40) {
  std::vector<double> k;
  if (a <= 0.0) return {1.0};
  const double x = a;  // I_m(2a) = sum_j a^(2j+m) / (j! (j+m)!)
  for (int m = 0; m <= rmax; ++m) {
    double term = exp(-2.0 * a);
    for (int i = 1; i <= m; ++i) term *= x / i;  // e^{-2a} a^m / m!
    double s = 0.0, t = term;
    for (int j = 0; j < 200; ++j) {
      s += t;
      t *= x * x / ((j + 1.0) * (j + 1.0 + m));
      if (t < 1e-30 * s) break;
    }
    if (m > 0 && s < tol) break;
    k.push_back(s);
  }
  return k;  // one side, k[0] at the centre
}

// ---------------------------------------------------------------------------
// Integrating-factor passes: out = sum_m k[|m|] in[. + m] along x, then along y
// (zero outside).  All taps in FP64 are 2 R + 1 ~ 27 operations per value on a
// unit that issues 1.7 per clock and SM: 50 us per pass of a 1023^2 field.  The
// taps |m| >= m0, whose sum is at most 2% (at 0.5 h^2 / kappa per step: |m| >=
// 3), are taken in float-float on the FP32 pipes instead: 2^-48 of 2% is below
// the rounding of the FP64 sum.  The values are split and put together again
// with integer operations (a conversion costs as much as an FP64 FMA).  A tile
// whose values leave FP32's exponent range takes every tap in FP64; a tile of
// zeros (most of R sigma) is skipped.  A 1023^2 step (the field,
// the sparse second one and the final sum): 32 us along x and 40 us along y; four
// FP64 passes and the sum took 4 x 51 + 10.
// ---------------------------------------------------------------------------
struct IFTaps {
  const double* k;    // R + 1
  const float2* kf;   // the same as (hi, lo)
  int R, m0;
};

__device__ __forceinline__ float2 split64(double v) {
  const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
  const int e = (int)(h >> 20 & 0x7ffu);
  const unsigned sg = h & 0x80000000u;
  float2 r = make_float2(0.f, 0.f);
  if (e > 896) {
    r.x = __uint_as_float(sg | (unsigned)(e - 896) << 23 | (h & 0xfffffu) << 3 | l >> 29);
    if (e > 948)  // the 29 bits below, in units of 2^(e - 1075)
      r.y = (float)(int)(l & 0x1fffffffu) * __uint_as_float(sg | (unsigned)(e - 948) << 23);
  }
  return r;
}
__device__ __forceinline__ float2 split64(float v) { return make_float2(v, 0.f); }

// stages one value; returns its magnitude bits for the tile's range
__device__ __forceinline__ unsigned stage_value(double v, float2 f, double* d, float2* s) {
  *d = v;
  *s = f;
  return (unsigned)__double2hiint(v) & 0x7fffffffu;
}

// what the tile's largest magnitude allows: in float-float from 2^-46 on, where
// what split64 drops of values below 2^-74 (2^-98, times 2% of far taps) stays
// under 2^-53 of it
enum { IF_ZERO = 0, IF_SPLIT = 1, IF_FP64 = 2 };
__device__ __forceinline__ int tile_mode(unsigned mag, unsigned low, unsigned* red) {
  if (threadIdx.x == 0) red[0] = red[1] = 0u;
  __syncthreads();
  mag = __reduce_max_sync(0xffffffffu, mag);
  low = __reduce_max_sync(0xffffffffu, low);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(red, mag);
    atomicMax(red + 1, low);
  }
  __syncthreads();
  const unsigned top = red[0] >> 20, any = red[0] | red[1];
  return any == 0u ? IF_ZERO : top >= 977u && top <= 1143u ? IF_SPLIT : IF_FP64;
}

// one output: centre index at, tap distance step
__device__ __forceinline__ double if_value(const double* d, const float2* f, int at, int step, const double* k,
                                           const float2* kf, int R, int m0, int mode) {
  double acc = k[0] * d[at];
  const int near = mode == IF_SPLIT ? min(m0 - 1, R) : R;
  for (int m = 1; m <= near; ++m) {
    acc = fma(k[m], d[at - m * step], acc);
    acc = fma(k[m], d[at + m * step], acc);
  }
  if (mode != IF_SPLIT) return acc;
  FF a{0.f, 0.f}, b{0.f, 0.f};
#pragma unroll 4
  for (int m = m0; m <= R; ++m) {
    const float2 c = kf[m], u = f[at - m * step], v = f[at + m * step];
    ff_fma(a, c.x, c.y, u.x, u.y);
    ff_fma(b, c.x, c.y, v.x, v.y);
  }
  a = ff_add(a, b);
  return acc + (widen(a.hi) + widen(a.lo));
}

constexpr int IF_T = 256;
constexpr int IFX_C = 128, IFX_R = 8;   // x pass: columns and rows of a tile
constexpr int IFY_C = 32, IFY_R = 32;   // y pass
constexpr int IF_RMAX = 40;

// taps into shared memory behind the tile
__device__ __forceinline__ void stage_taps(const IFTaps& t, double* k, float2* kf) {
  for (int m = threadIdx.x; m <= t.R; m += IF_T) {
    k[m] = t.k[m];
    kf[m] = t.kf[m];
  }
}

// x pass of up to two fields (blockIdx.z)
template <typename T>
__global__ void __launch_bounds__(IF_T) k_if_x(int n1, int n2, IFTaps t0, const T* __restrict__ in0, T* __restrict__ out0,
                                               IFTaps t1, const T* __restrict__ in1, T* __restrict__ out1) {
  extern __shared__ __align__(16) double if_sm[];
  __shared__ unsigned red[2];
  __shared__ double k[IF_RMAX + 1];
  __shared__ float2 kf[IF_RMAX + 1];
  const IFTaps t = blockIdx.z ? t1 : t0;
  const T* __restrict__ in = blockIdx.z ? in1 : in0;
  T* __restrict__ out = blockIdx.z ? out1 : out0;
  const int W = IFX_C + 2 * t.R, x0 = blockIdx.x * IFX_C, y0 = blockIdx.y * IFX_R;
  double* d = if_sm;
  float2* f = reinterpret_cast<float2*>(d + W * IFX_R);
  stage_taps(t, k, kf);
  unsigned mag = 0u, low = 0u;
  for (int q = threadIdx.x; q < W * IFX_R; q += IF_T) {
    const int r = q / W, i = x0 + q - r * W - t.R, j = y0 + r;
    const T v = i >= 0 && i < n1 && j < n2 ? in[(size_t)j * n1 + i] : (T)0;
    mag = max(mag, stage_value((double)v, split64(v), d + q, f + q));
    low |= (unsigned)__double2loint((double)v);
  }
  const int mode = tile_mode(mag, low, red);
  const int c = threadIdx.x % IFX_C, i = x0 + c;
  if (i >= n1) return;
  for (int r = threadIdx.x / IFX_C; r < IFX_R && y0 + r < n2; r += IF_T / IFX_C)
    out[(size_t)(y0 + r) * n1 + i] =
        mode == IF_ZERO ? (T)0 : (T)if_value(d, f, r * W + c + t.R, 1, k, kf, t.R, t.m0, mode);
}

// y pass: out = IFy_0 in0 (+ c1 IFy_1 in1 + c2 add2 + add3, where given)
template <typename T>
__global__ void __launch_bounds__(IF_T) k_if_y(int n1, int n2, IFTaps t0, const T* __restrict__ in0, IFTaps t1, double c1,
                                               const T* __restrict__ in1, double c2, const T* __restrict__ add2,
                                               const T* __restrict__ add3, T* __restrict__ out) {
  extern __shared__ __align__(16) double if_sm[];
  __shared__ unsigned red[2];
  __shared__ double k[IF_RMAX + 1];
  __shared__ float2 kf[IF_RMAX + 1];
  constexpr int PER = IFY_R * IFY_C / IF_T;
  const int x0 = blockIdx.x * IFY_C, y0 = blockIdx.y * IFY_R, c = threadIdx.x % IFY_C, r0 = threadIdx.x / IFY_C;
  const int i = x0 + c;
  double acc[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) acc[q] = 0.0;
  for (int fld = 0; fld < (in1 ? 2 : 1); ++fld) {
    const IFTaps t = fld ? t1 : t0;
    const T* __restrict__ in = fld ? in1 : in0;
    const int rows = IFY_R + 2 * t.R;
    double* d = if_sm;
    float2* f = reinterpret_cast<float2*>(d + rows * IFY_C);
    stage_taps(t, k, kf);
    unsigned mag = 0u, low = 0u;
    for (int q = threadIdx.x; q < rows * IFY_C; q += IF_T) {
      const int j = y0 + q / IFY_C - t.R;
      const T v = i < n1 && j >= 0 && j < n2 ? in[(size_t)j * n1 + i] : (T)0;
      mag = max(mag, stage_value((double)v, split64(v), d + q, f + q));
      low |= (unsigned)__double2loint((double)v);
    }
    const int mode = tile_mode(mag, low, red);
    if (mode != IF_ZERO && i < n1) {
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int r = r0 + q * (IF_T / IFY_C);
        if (y0 + r >= n2) continue;
        const double v = if_value(d, f, (r + t.R) * IFY_C + c, IFY_C, k, kf, t.R, t.m0, mode);
        acc[q] = fld ? fma(c1, v, acc[q]) : v;
      }
    }
    __syncthreads();
  }
  if (i >= n1) return;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int j = y0 + r0 + q * (IF_T / IFY_C);
    if (j >= n2) continue;
    const size_t at = (size_t)j * n1 + i;
    double v = acc[q];
    if (add2) v = fma(c2, (double)add2[at], v) + (double)add3[at];
    out[at] = (T)v;
  }
}

// smeared-window gather: out_k = sum_{jj,ii} wy[k][jj] wx[k][ii] T[by+jj][bx+ii]
// one warp per point; two window sets (two integrating-factor arguments)
template <typename T>
__global__ void k_conv_gather2(int N, int n1, int n2, const T* __restrict__ f, int L0, const int* __restrict__ bx0,
                               const int* __restrict__ by0, const double* __restrict__ wx0,
                               const double* __restrict__ wy0, double* __restrict__ out0, int L1,
                               const int* __restrict__ bx1, const int* __restrict__ by1,
                               const double* __restrict__ wx1, const double* __restrict__ wy1,
                               double* __restrict__ out1) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= 2 * N) return;
  const int set = warp >= N ? 1 : 0;
  const int k = warp - set * N;
  const int L = set ? L1 : L0;
  const int b0 = set ? bx1[k] : bx0[k];
  const int e0 = set ? by1[k] : by0[k];
  const double* wx = (set ? wx1 : wx0) + (size_t)k * L;
  const double* wy = (set ? wy1 : wy0) + (size_t)k * L;
  // a lane keeps its columns (one, or three at most: L <= 84) and sums over the
  // rows, eight rows' loads in flight; the column weight comes last
  double acc = 0.0;
  for (int ii = lane; ii < L; ii += 32) {
    const int i = b0 + ii;
    if ((unsigned)i >= (unsigned)n1) continue;
    double col = 0.0;
#pragma unroll 8
    for (int jj = 0; jj < L; ++jj) {
      const int j = e0 + jj;
      if ((unsigned)j < (unsigned)n2) col = fma(wy[jj], (double)f[(size_t)j * n1 + i], col);
    }
    acc = fma(wx[ii], col, acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0) (set ? out1 : out0)[k] = acc;
}

// Stage right-hand sides, a warp per point: rhs = (avg - (g + c0 v0 + c1 S x +
// c2 v2)) / denom, S a stage matrix in CSR (rowptr null: without its term and
// the next)
__global__ void k_stage_rhs(int n, const double* __restrict__ avg, const double* __restrict__ g, double c0,
                            const double* __restrict__ v0, double c1, const int* __restrict__ rowptr,
                            const int* __restrict__ col, const float* __restrict__ vhi, const float* __restrict__ vlo,
                            const double* __restrict__ x, double c2, const double* __restrict__ v2, double inv_denom,
                            double* __restrict__ rhs) {
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (k >= n) return;
  double q = 0.0;
  if (rowptr) {
    for (int e = rowptr[k] + lane; e < rowptr[k + 1]; e += 32) q += ((double)vhi[e] + (double)vlo[e]) * x[col[e]];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_down_sync(0xffffffffu, q, o);
  }
  if (lane == 0) {
    double s = g[k] + c0 * v0[k];
    if (rowptr) {
      s += c1 * q;
      s += c2 * v2[k];
    }
    rhs[k] = (avg[k] - s) * inv_denom;
  }
}

}  // namespace

}  // namespace ilm

using namespace ilm;

constexpr int HEAT_MAX_POINTS = 4688;  // unknowns of a stage solve

struct ilm_heat_s {
  ilm_cache_s* c = nullptr;
  double kappa = 1.0, dt = 0.0;
  double a21 = 1.0 / 3.0, a31 = -1.0, a32 = 2.0, b1 = 0.0, b2 = 0.75, b3 = 0.25;
  double tol = 1e-10;
  int maxiter = 2000;
  int n1 = 0, n2 = 0;
  // integrating-factor taps for a * (1/3, 2/3, 1)
  int R[3] = {0, 0, 0};
  DevBuf kt[3], ktf[3];
  int m0[3] = {1, 1, 1};
  // smeared gather windows for a/3 (set 0) and a (set 1)
  int L[2] = {0, 0};
  DevBuf gbx[2], gby[2], gwx[2], gwy[2];
  // sparse stage Schur complements: 0 -> a/3, 1 -> 2a/3, 2 -> a, 3 -> 0
  DevBuf rowptr[4], colidx[4], vhi[4], vlo[4];
  size_t nnz[4] = {0, 0, 0, 0};
  DevBuf e[4], avg64, cfield;
  DevBuf g1, g3, rhs, sig[3], sig_t;
  DevBuf tmp[4];
  DevBuf cgs, iters, relres;
  CG64Inverse inv[3];             // FP32 inverses of the three stage systems
  int max_row[4] = {0, 0, 0, 0};  // most entries of a row
  long long total_iters = 0;
  int last_iters[3] = {0, 0, 0};
};

namespace {

int upd(DevBuf& b, const void* h, size_t bytes) {
  ILM_TRY(b.alloc(std::max<size_t>(bytes, 8)));
  if (bytes) ILM_CHECK_CUDA(cudaMemcpy(b.p, h, bytes, cudaMemcpyHostToDevice));
  return ILM_OK;
}

IFTaps taps_of(const ilm_heat_s* H, int which) {
  return IFTaps{H->kt[which].as<double>(), H->ktf[which].as<float2>(), H->R[which], H->m0[which]};
}

// out = exp(a_0 L) in0 (+ c1 exp(a_1 L) in1 + c2 add2 + add3); tmp0, tmp1: the fields after their x pass
template <typename T>
int apply_if(const ilm_heat_s* H, int w0, const void* in0, void* tmp0, int w1, double c1, const void* in1, void* tmp1,
             double c2, const void* add2, const void* add3, void* out, cudaStream_t st) {
  const IFTaps t0 = taps_of(H, w0), t1 = in1 ? taps_of(H, w1) : t0;
  const int R = std::max(t0.R, t1.R), n1 = H->n1, n2 = H->n2;
  const size_t sx = (size_t)(IFX_C + 2 * R) * IFX_R * 16, sy = (size_t)(IFY_R + 2 * R) * IFY_C * 16;
  ILM_CHECK_CUDA(cudaFuncSetAttribute(k_if_x<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
  ILM_CHECK_CUDA(cudaFuncSetAttribute(k_if_y<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
  k_if_x<T><<<dim3((n1 + IFX_C - 1) / IFX_C, (n2 + IFX_R - 1) / IFX_R, in1 ? 2 : 1), IF_T, sx, st>>>(
      n1, n2, t0, static_cast<const T*>(in0), static_cast<T*>(tmp0), t1, static_cast<const T*>(in1),
      static_cast<T*>(tmp1));
  ILM_CHECK_LAUNCH();
  k_if_y<T><<<dim3((n1 + IFY_C - 1) / IFY_C, (n2 + IFY_R - 1) / IFY_R), IF_T, sy, st>>>(
      n1, n2, t0, static_cast<const T*>(tmp0), t1, c1, static_cast<const T*>(in1 ? tmp1 : nullptr), c2,
      static_cast<const T*>(add2), static_cast<const T*>(add3), static_cast<T*>(out));
  ILM_CHECK_LAUNCH();
  return ILM_OK;
}

// sparse S_a = E exp(aL) R on Nodes{Primal}: S_kl = (ds_l/h^2) X_kl Y_kl with X_kl the
// x-window of k smeared by the heat kernel, correlated with l's x-window.
int build_sparse_schur(ilm_heat_s* H, const std::vector<double>& taps, int slot) {
  ilm_cache_s* c = H->c;
  const int N = c->npts;
  const int R = (int)taps.size() - 1;
  const int reach = 2 * R + NTAP;  // |bx_k - bx_l| < reach for a nonzero X_kl
  const std::vector<int>& bx = c->hbx[0];
  const std::vector<int>& by = c->hby[0];
  const std::vector<double>& wx = c->hwx[0];
  const std::vector<double>& wy = c->hwy[0];
  auto kval = [&](int m) { m = m < 0 ? -m : m; return m <= R ? taps[m] : 0.0; };
  // smeared windows (length NTAP + 2R, base bx - R)
  const int Ls = NTAP + 2 * R;
  std::vector<double> sx((size_t)N * Ls, 0.0), sy((size_t)N * Ls, 0.0);
  for (int k = 0; k < N; ++k)
    for (int t = 0; t < NTAP; ++t)
      for (int m = -R; m <= R; ++m) {
        sx[(size_t)k * Ls + t + m + R] += wx[(size_t)k * NTAP + t] * kval(m);
        sy[(size_t)k * Ls + t + m + R] += wy[(size_t)k * NTAP + t] * kval(m);
      }
  // spatial hash of points by window base
  const int B = std::max(reach, 1);
  std::unordered_map<long long, std::vector<int>> cells;
  auto key = [](int a, int b) { return ((long long)a << 32) ^ (unsigned int)b; };
  auto fdiv = [](int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); };
  for (int k = 0; k < N; ++k) cells[key(fdiv(bx[k], B), fdiv(by[k], B))].push_back(k);
  std::vector<int> rp(N + 1, 0), ci;
  std::vector<float> vh, vl;
  const double ih2 = 1.0 / (c->h * c->h);
  std::vector<int> nb;
  for (int k = 0; k < N; ++k) {
    nb.clear();
    const int cx = fdiv(bx[k], B), cy = fdiv(by[k], B);
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        auto it = cells.find(key(cx + dx, cy + dy));
        if (it == cells.end()) continue;
        for (int l : it->second)
          if (std::abs(bx[k] - bx[l]) < reach && std::abs(by[k] - by[l]) < reach) nb.push_back(l);
      }
    std::sort(nb.begin(), nb.end());
    for (int l : nb) {
      // X_kl = sum_u wx_l[u] * sx_k[(bx_l + u) - (bx_k - R)]
      double X = 0.0, Y = 0.0;
      for (int u = 0; u < NTAP; ++u) {
        const int ix = bx[l] + u - (bx[k] - R);
        if (ix >= 0 && ix < Ls) X += wx[(size_t)l * NTAP + u] * sx[(size_t)k * Ls + ix];
        const int iy = by[l] + u - (by[k] - R);
        if (iy >= 0 && iy < Ls) Y += wy[(size_t)l * NTAP + u] * sy[(size_t)k * Ls + iy];
      }
      const double v = c->hds[l] * ih2 * X * Y;
      if (v == 0.0) continue;
      ci.push_back(l);
      const float h = (float)v;
      vh.push_back(h);
      vl.push_back((float)(v - (double)h));
    }
    rp[k + 1] = (int)ci.size();
  }
  H->nnz[slot] = ci.size();
  for (int k = 0; k < N; ++k) H->max_row[slot] = std::max(H->max_row[slot], rp[k + 1] - rp[k]);
  ILM_TRY(upd(H->rowptr[slot], rp.data(), rp.size() * sizeof(int)));
  ILM_TRY(upd(H->colidx[slot], ci.data(), ci.size() * sizeof(int)));
  ILM_TRY(upd(H->vhi[slot], vh.data(), vh.size() * sizeof(float)));
  ILM_TRY(upd(H->vlo[slot], vl.data(), vl.size() * sizeof(float)));
  return ILM_OK;
}

// smeared gather windows on Nodes{Primal} for one integrating-factor argument
int build_gather_windows(ilm_heat_s* H, const std::vector<double>& taps, int set) {
  ilm_cache_s* c = H->c;
  const int N = c->npts;
  const int R = (int)taps.size() - 1;
  const int Ls = NTAP + 2 * R;
  std::vector<int> bx(N), by(N);
  std::vector<double> sx((size_t)N * Ls, 0.0), sy((size_t)N * Ls, 0.0);
  for (int k = 0; k < N; ++k) {
    bx[k] = c->hbx[0][k] - R;
    by[k] = c->hby[0][k] - R;
    for (int t = 0; t < NTAP; ++t)
      for (int m = -R; m <= R; ++m) {
        const double km = taps[std::abs(m)];
        sx[(size_t)k * Ls + t + m + R] += c->hwx[0][(size_t)k * NTAP + t] * km;
        sy[(size_t)k * Ls + t + m + R] += c->hwy[0][(size_t)k * NTAP + t] * km;
      }
  }
  H->L[set] = Ls;
  ILM_TRY(upd(H->gbx[set], bx.data(), N * sizeof(int)));
  ILM_TRY(upd(H->gby[set], by.data(), N * sizeof(int)));
  ILM_TRY(upd(H->gwx[set], sx.data(), sx.size() * sizeof(double)));
  ILM_TRY(upd(H->gwy[set], sy.data(), sy.size() * sizeof(double)));
  return ILM_OK;
}

// the system S sigma = rhs of stage s (0: a/3, 1: 2a/3, 2: the final update)
CG64Problem stage_problem(ilm_heat_s* H, int s) {
  constexpr int slot[3] = {0, 1, 3};
  const int m = slot[s], N = H->c->npts;
  CG64Problem P;
  P.rowptr = H->rowptr[m].as<int>();
  P.colidx = H->colidx[m].as<int>();
  P.vhi = H->vhi[m].as<float>();
  P.vlo = H->vlo[m].as<float>();
  P.max_row_nnz = H->max_row[m];
  P.w = H->c->ds64.as<double>();
  P.n = N;
  P.maxiter = H->maxiter;
  P.tol = H->tol;
  P.refresh = 50;
  P.stall = 8;
  return P;
}

// from the last step's sigma
int run_cg(ilm_heat_s* H, int s, cudaStream_t st) {
  CG64Problem P = stage_problem(H, s);
  if (P.n > HEAT_MAX_POINTS) {
    set_error("heat: %d points exceed the stage solver's limit of %d", P.n, HEAT_MAX_POINTS);
    return ILM_ERR_SIZE_LIMIT;
  }
  P.b = H->rhs.as<double>() + (size_t)s * P.n;
  P.x = H->sig[s].as<double>();
  P.x0 = H->sig[s].as<double>();
  P.iters = H->iters.as<int>() + s;
  P.relres = H->relres.as<double>() + s;
  P.timeout = H->iters.as<int>() + 3;
  if (H->inv[s].ready) H->inv[s].attach(&P);
  return launch_cg64(P, H->cgs.p, st);
}

}  // namespace

extern "C" {

int ilm_heat_create(ilm_cache_t c, double kappa, double dt, const double* tb_plus, const double* tb_minus,
                    double tol, int maxiter, ilm_heat_t* out) {
  if (c) ILM_TRY(cache_sync_host(c));  // host windows used below
  ILM_REQUIRE(c && out && tb_plus && tb_minus, "heat: null argument");
  ILM_REQUIRE(c->kind == ILM_CACHE_SCALAR, "heat: scalar cache required");
  ILM_REQUIRE(c->scaling == ILM_GRID_SCALING, "heat: GridScaling cache required");
  ILM_REQUIRE(c->npts > 0, "heat: the cache has no surface points");
  ILM_REQUIRE(kappa > 0 && dt > 0 && tol > 0 && maxiter > 0, "heat: bad kappa / dt / tol / maxiter");
  const double af = kappa * dt / (c->h * c->h);
  ILM_REQUIRE(af <= 4.0, "heat: kappa dt / h^2 = %g too large for the integrating-factor stencil", af);
  auto* H = new (std::nothrow) ilm_heat_s();
  if (!H) return ILM_ERR_NO_MEMORY;
  std::unique_ptr<ilm_heat_s> guard(H);
  H->c = c;
  H->kappa = kappa;
  H->dt = dt;
  H->tol = tol;
  H->maxiter = maxiter;
  const ilm::Shape2 sh = c->grid.shape(PC_P);
  H->n1 = sh.n1;
  H->n2 = sh.n2;
  const int N = c->npts;
  const size_t np = sh.numel();
  const size_t es = c->dtype == ILM_F64 ? 8 : 4;
  const double frac[3] = {1.0 / 3.0, 2.0 / 3.0, 1.0};
  std::vector<double> taps[3];
  for (int w = 0; w < 3; ++w) {
    taps[w] = heat_kernel_taps(af * frac[w]);
    H->R[w] = (int)taps[w].size() - 1;
    ILM_TRY(upd(H->kt[w], taps[w].data(), taps[w].size() * sizeof(double)));
    std::vector<float> tf(2 * taps[w].size());
    double far = 0.0;
    H->m0[w] = H->R[w] + 1;  // the taps from m0 on add up to at most 2% (both sides)
    for (int m = H->R[w]; m >= 0; --m) {
      tf[2 * m] = (float)taps[w][m];
      tf[2 * m + 1] = (float)(taps[w][m] - (double)tf[2 * m]);
      far += 2.0 * taps[w][m];
      if (m > 0 && far <= 0.02) H->m0[w] = m;
    }
    ILM_TRY(upd(H->ktf[w], tf.data(), tf.size() * sizeof(float)));
  }
  ILM_TRY(build_gather_windows(H, taps[0], 0));
  ILM_TRY(build_gather_windows(H, taps[2], 1));
  const std::vector<double> delta{1.0};
  ILM_TRY(build_sparse_schur(H, taps[0], 0));
  ILM_TRY(build_sparse_schur(H, taps[1], 1));
  ILM_TRY(build_sparse_schur(H, taps[2], 2));
  ILM_TRY(build_sparse_schur(H, delta, 3));
  // surface data, r1 = -kappa D_s[T] and its point images e_a = E exp(aL) r1
  std::vector<double> avg(N), jump(N);
  for (int k = 0; k < N; ++k) {
    avg[k] = 0.5 * (tb_plus[k] + tb_minus[k]);
    jump[k] = -kappa * (tb_plus[k] - tb_minus[k]);
  }
  ILM_TRY(upd(H->avg64, avg.data(), N * sizeof(double)));
  for (int t = 0; t < 4; ++t) ILM_TRY(H->tmp[t].alloc(np * es));
  DevBuf jd, pt;
  ILM_TRY(jd.alloc((size_t)N * es));
  ILM_TRY(pt.alloc((size_t)N * es));
  if (c->dtype == ILM_F64) {
    ILM_CHECK_CUDA(cudaMemcpy(jd.p, jump.data(), N * 8, cudaMemcpyHostToDevice));
  } else {
    std::vector<float> jf(jump.begin(), jump.end());
    ILM_CHECK_CUDA(cudaMemcpy(jd.p, jf.data(), N * 4, cudaMemcpyHostToDevice));
  }
  void* r1 = H->tmp[0].p;
  ILM_TRY(ilm_surface_divergence(c, jd.p, r1, nullptr));
  ILM_TRY(H->cfield.alloc(np * es));
  for (int t = 0; t < 4; ++t) ILM_TRY(H->e[t].alloc((size_t)N * 8));
  for (int w = 0; w < 3; ++w) {
    ILM_TRY((c->dtype == ILM_F64 ? apply_if<double> : apply_if<float>)(H, w, r1, H->tmp[1].p, 0, 0.0, nullptr, nullptr,
                                                                       0.0, nullptr, nullptr, H->tmp[2].p, nullptr));
    ILM_TRY(ilm_interpolate(c, ILM_NODES_PRIMAL, H->tmp[2].p, pt.p, nullptr));
    ILM_TRY(st_convert(N, c->dtype, pt.p, ILM_F64, H->e[w].p, nullptr));
    if (w == 1) {  // cfield = dt b2 exp(2a/3 L) r1 + dt b3 r1   (b1 = 0)
      ILM_TRY(st_axpby(np, c->dtype, dt * H->b2, H->tmp[2].p, dt * H->b3, r1, H->cfield.p, nullptr));
    }
  }
  ILM_TRY(ilm_interpolate(c, ILM_NODES_PRIMAL, r1, pt.p, nullptr));
  ILM_TRY(st_convert(N, c->dtype, pt.p, ILM_F64, H->e[3].p, nullptr));
  // work vectors and CG parameter records (stage 2: S_{a/3}; stage 3: S_{2a/3}; final: S_0)
  ILM_TRY(H->g1.alloc((size_t)N * 8));
  ILM_TRY(H->g3.alloc((size_t)N * 8));
  ILM_TRY(H->rhs.alloc((size_t)N * 8 * 3));
  for (int s = 0; s < 3; ++s) {
    ILM_TRY(H->sig[s].alloc((size_t)N * 8));
    ILM_CHECK_CUDA(cudaMemset(H->sig[s].p, 0, (size_t)N * 8));
  }
  ILM_TRY(H->sig_t.alloc((size_t)N * es));
  ILM_TRY(H->iters.alloc(4 * sizeof(int)));  // and the solver's time-out flag
  ILM_CHECK_CUDA(cudaMemset(H->iters.p, 0, 4 * sizeof(int)));
  ILM_TRY(H->relres.alloc(3 * sizeof(double)));
  ILM_TRY(H->cgs.alloc(cg64_scratch_bytes(N)));
  DevBuf tmp;
  if (N <= HEAT_MAX_POINTS)
    for (int s = 0; s < 3; ++s) ILM_TRY(cg64_inverse(&H->inv[s], &tmp, stage_problem(H, s), nullptr));
  ILM_CHECK_CUDA(cudaDeviceSynchronize());
  *out = guard.release();
  return ILM_OK;
}

int ilm_heat_destroy(ilm_heat_t h) {
  delete h;
  return ILM_OK;
}

int ilm_heat_advance(ilm_heat_t H, void* T, void* sigma_out, int nsteps, ilm_stream_t stream) {
  ILM_REQUIRE(H && T && nsteps >= 0, "heat_advance: bad arguments");
  ilm_cache_s* c = H->c;
  cudaStream_t st = as_stream(stream);
  const int N = c->npts;
  const double dt = H->dt;
  const int wb = (2 * N * 32 + 255) / 256;
  const int sb = (N * 32 + 255) / 256;
  double* rhs = H->rhs.as<double>();
  for (int step = 0; step < nsteps; ++step) {
    // point images of the current field: g1 = E exp(a/3 L) T, g3 = E exp(a L) T
    if (c->dtype == ILM_F64)
      k_conv_gather2<double><<<wb, 256, 0, st>>>(N, H->n1, H->n2, static_cast<const double*>(T), H->L[0],
                                                  H->gbx[0].as<int>(), H->gby[0].as<int>(), H->gwx[0].as<double>(),
                                                  H->gwy[0].as<double>(), H->g1.as<double>(), H->L[1],
                                                  H->gbx[1].as<int>(), H->gby[1].as<int>(), H->gwx[1].as<double>(),
                                                  H->gwy[1].as<double>(), H->g3.as<double>());
    else
      k_conv_gather2<float><<<wb, 256, 0, st>>>(N, H->n1, H->n2, static_cast<const float*>(T), H->L[0],
                                                 H->gbx[0].as<int>(), H->gby[0].as<int>(), H->gwx[0].as<double>(),
                                                 H->gwy[0].as<double>(), H->g1.as<double>(), H->L[1],
                                                 H->gbx[1].as<int>(), H->gby[1].as<int>(), H->gwx[1].as<double>(),
                                                 H->gwy[1].as<double>(), H->g3.as<double>());
    ILM_CHECK_LAUNCH();
    // stage 2: S_{a/3} sigma1 = (avg - g1 - dt a21 e_{a/3}) / (dt a21)
    k_stage_rhs<<<sb, 256, 0, st>>>(N, H->avg64.as<double>(), H->g1.as<double>(), dt * H->a21, H->e[0].as<double>(),
                                     0.0, nullptr, nullptr, nullptr, nullptr, nullptr, 0.0, nullptr,
                                     1.0 / (dt * H->a21), rhs);
    ILM_CHECK_LAUNCH();
    ILM_TRY(run_cg(H, 0, st));
    // stage 3: S_{2a/3} sigma2 = (avg - [g3 + dt a31 (e_a + S_a sigma1) + dt a32 e_{2a/3}]) / (dt a32)
    k_stage_rhs<<<sb, 256, 0, st>>>(N, H->avg64.as<double>(), H->g3.as<double>(), dt * H->a31, H->e[2].as<double>(),
                                     dt * H->a31, H->rowptr[2].as<int>(), H->colidx[2].as<int>(),
                                     H->vhi[2].as<float>(), H->vlo[2].as<float>(), H->sig[0].as<double>(), dt * H->a32,
                                     H->e[1].as<double>(), 1.0 / (dt * H->a32), rhs + N);
    ILM_CHECK_LAUNCH();
    ILM_TRY(run_cg(H, 1, st));
    // final: S_0 sigma3 = (avg - [g3 + dt b2 (e_{2a/3} + S_{2a/3} sigma2) + dt b3 e_0]) / (dt b3)   (b1 = 0)
    k_stage_rhs<<<sb, 256, 0, st>>>(N, H->avg64.as<double>(), H->g3.as<double>(), dt * H->b2, H->e[1].as<double>(),
                                     dt * H->b2, H->rowptr[1].as<int>(), H->colidx[1].as<int>(),
                                     H->vhi[1].as<float>(), H->vlo[1].as<float>(), H->sig[1].as<double>(), dt * H->b3,
                                     H->e[3].as<double>(), 1.0 / (dt * H->b3), rhs + 2 * N);
    ILM_CHECK_LAUNCH();
    ILM_TRY(run_cg(H, 2, st));
    // grid: T <- exp(aL) T + dt b2 exp(2a/3 L) R sigma2 + dt b3 R sigma3 + cfield
    for (int k = 1; k <= 2; ++k) {
      const void* sig = H->sig[k].p;
      if (c->dtype != ILM_F64) {
        ILM_TRY(st_convert(N, ILM_F64, sig, c->dtype, H->sig_t.p, st));
        sig = H->sig_t.p;
      }
      ILM_TRY(ilm_regularize(c, ILM_NODES_PRIMAL, sig, H->tmp[k + 1].p, st));
    }
    ILM_TRY((c->dtype == ILM_F64 ? apply_if<double> : apply_if<float>)(H, 2, T, H->tmp[0].p, 1, dt * H->b2, H->tmp[2].p,
                                                                       H->tmp[1].p, dt * H->b3, H->tmp[3].p,
                                                                       H->cfield.p, T, st));
  }
  if (sigma_out) {  // the reference's constraint force enters as -R sigma
    ILM_TRY(st_convert(N, ILM_F64, H->sig[2].p, c->dtype, sigma_out, st));
    ILM_TRY(st_affine(N, c->dtype, -1.0, sigma_out, 0.0, sigma_out, st));
  }
  if (nsteps > 0) {
    int it[4];
    ILM_CHECK_CUDA(cudaMemcpyAsync(it, H->iters.p, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
    ILM_CHECK_CUDA(cudaStreamSynchronize(st));
    if (it[3]) {
      ILM_CHECK_CUDA(cudaMemset(H->iters.as<int>() + 3, 0, sizeof(int)));
      set_error("heat: a stage solve's wait for the other CTAs ran out");
      return ILM_ERR_TIMEOUT;
    }
    for (int s = 0; s < 3; ++s) H->last_iters[s] = it[s];
  }
  return ILM_OK;
}

int ilm_heat_info(ilm_heat_t H, int* last_iters, double* last_relres, size_t* nnz) {
  ILM_REQUIRE(H, "null heat integrator");
  if (last_iters) ILM_CHECK_CUDA(cudaMemcpy(last_iters, H->iters.p, 3 * sizeof(int), cudaMemcpyDeviceToHost));
  if (last_relres) ILM_CHECK_CUDA(cudaMemcpy(last_relres, H->relres.p, 3 * sizeof(double), cudaMemcpyDeviceToHost));
  if (nnz)
    for (int s = 0; s < 4; ++s) nnz[s] = H->nnz[s];
  return ILM_OK;
}

}  // extern "C"
