// Schur complements of the immersed-layer saddle-point systems and their
// on-device Krylov solve.
//
// The reference builds each dense Schur complement column by column, with one
// regularize! + inverse_laplacian! (an FFT convolution of the whole grid) +
// interpolate! per column (src/matrix_operators.jl:9-244), then solves it with
// a dense LU on every call (test/literate/problems.jl:291, neumann.jl:123).
//
// Here every entry is evaluated directly from the lattice Green's function:
// the interpolation-side and regularization-side operators of point k are
// short separable stencils U_k (4 or 5 taps per direction, up to two terms),
// and since L^{-1} is the exact linear convolution with G,
//     (U L^{-1} V^T)_{kl} = (1/factor) sum_{a,b} U_k(a) G(a-b) V_l(b)
//                         = (1/factor) sum_{dx,dy} Cx(dx) Cy(dy) G(D + (dx,dy)),
// with Cx, Cy the 1-D correlations of the two stencils (7 to 9 values each) and D
// the offset of the stencil bases.  This is O(N^2 * 49) to O(N^2 * 288) FP64 work
// instead of O(N * P^2 log P), and gives the same matrix (up to FP64 rounding) provided
// every stencil stays clear of the grid's ghost layer.
//
// The solve (ilm_cg64.cu) refines an FP32 inverse with FP64 residuals and goes
// on by CG in the ds-weighted inner product (the matrices are M*diag(w) with M
// symmetric) in FP64 where that stalls: an FP32 matvec in the CG loses the Krylov
// convergence on these ill-conditioned (cond ~ 1e4-1e5) and, for the
// Dirichlet problem, indefinite (one negative eigenvalue) systems.
// Convergence is declared on the FP64 residual ||b - A x||_2 <= tol ||b||_2.
#include <math.h>
#include <stddef.h>

#include <algorithm>

#include "ilm_internal.cuh"

namespace ilm {

constexpr int FW = 5;  // functional window width

struct Functional {
  // two separable terms: coef, x base, y base, 5 x-weights, 5 y-weights
  double coef[2];
  int xb[2], yb[2];
  double xw[2][FW], yw[2][FW];
  int nterm;
};

// The same functional with every weight split into a float-float (hi, lo)
// pair once per point, for the batched float-float builds (the split is an
// FP64 subtraction, which GB300 issues at a small fraction of its FP32 rate;
// split per point pair it was a large part of the build).  Written over the
// Functional buffers, so it is no larger.
struct alignas(8) FunctionalFF {
  float coef[2][2];
  float w[2];                  // the point's regularization weight ds (hi, lo)
  short xb[2], yb[2], nterm, pad_[3];  // grid base indices (|index| < 32768)
  float xw[2][FW][2], yw[2][FW][2];
};
static_assert(sizeof(FunctionalFF) <= sizeof(Functional), "FunctionalFF overlays Functional buffers");
static_assert(offsetof(FunctionalFF, xw) % 8 == 0 && offsetof(FunctionalFF, yw) % 8 == 0, "weight pairs are read as float2");

// Build the per-point functionals for one Schur kind.  side 0 = left
// (interpolation side, no ds weight), side 1 = right (regularization side).
__global__ void k_functionals(int N, int kind, const int* __restrict__ bxP, const int* __restrict__ bxD,
                              const int* __restrict__ byP, const int* __restrict__ byD,
                              const double* __restrict__ wxP, const double* __restrict__ wxD,
                              const double* __restrict__ wyP, const double* __restrict__ wyD,
                              const double* __restrict__ nx, const double* __restrict__ ny, double invh,
                              Functional* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
  Functional F;
  for (int p = 0; p < 2; ++p) {
    F.coef[p] = 0.0;
    F.xb[p] = F.yb[p] = 0;
    for (int t = 0; t < FW; ++t) F.xw[p][t] = F.yw[p][t] = 0.0;
  }
  const double* wxp = wxP + (size_t)k * NTAP;
  const double* wxd = wxD + (size_t)k * NTAP;
  const double* wyp = wyP + (size_t)k * NTAP;
  const double* wyd = wyD + (size_t)k * NTAP;
  auto at = [](const double* w, int t) { return (t >= 0 && t < NTAP) ? w[t] : 0.0; };
  if (kind == ILM_SCHUR_RTLINVR) {
    // plain E on Nodes{Primal}
    F.nterm = 1;
    F.coef[0] = 1.0;
    F.xb[0] = bxP[k];
    F.yb[0] = byP[k];
    for (int t = 0; t < NTAP; ++t) {
      F.xw[0][t] = wxp[t];
      F.yw[0][t] = wyp[t];
    }
  } else if (kind == ILM_SCHUR_CLINVCT) {
    // C_s on Nodes{Dual}: (n_x/h) [wxD (x) (wyP[t-1]-wyP[t])] + (n_y/h) [(wxP[t]-wxP[t-1]) (x) wyD]
    F.nterm = 2;
    F.coef[0] = nx[k] * invh;
    F.xb[0] = bxD[k];
    F.yb[0] = byP[k];
    for (int t = 0; t < FW; ++t) {
      F.xw[0][t] = at(wxd, t);
      F.yw[0][t] = at(wyp, t - 1) - at(wyp, t);
    }
    F.coef[1] = ny[k] * invh;
    F.xb[1] = bxP[k];
    F.yb[1] = byD[k];
    for (int t = 0; t < FW; ++t) {
      F.xw[1][t] = at(wxp, t) - at(wxp, t - 1);
      F.yw[1][t] = at(wyd, t);
    }
  } else {  // ILM_SCHUR_GLINVD: D_s functional on Nodes{Primal}
    F.nterm = 2;
    F.coef[0] = nx[k] * invh;
    F.xb[0] = bxD[k] - 1;
    F.yb[0] = byP[k];
    for (int t = 0; t < FW; ++t) {
      F.xw[0][t] = at(wxd, t) - at(wxd, t - 1);
      F.yw[0][t] = at(wyp, t);
    }
    F.coef[1] = ny[k] * invh;
    F.xb[1] = bxP[k];
    F.yb[1] = byD[k] - 1;
    for (int t = 0; t < FW; ++t) {
      F.xw[1][t] = at(wxp, t);
      F.yw[1][t] = at(wyd, t) - at(wyd, t - 1);
    }
  }
  out[k] = F;
}

// A term's weights have NTAP entries along one axis (both, for plain
// interpolation) and FW along the other, which holds the difference.  Taken by
// the short axis of k's term, a pair of terms is one of two shapes (G depends
// on the distances alone, and is symmetric in them): l short on the same axis,
// or on the other.
__device__ __forceinline__ bool short_in_x(int kind, int p) {
  return kind == ILM_SCHUR_GLINVD ? p == 1 : p == 0;
}

// tile (ti, tj), ti <= tj, of the upper triangle's tile t in row-major order
__device__ __forceinline__ void triangle_tile(int t, int nt, int* ti_, int* tj_) {
  // tile row of triangle index t (FP32 estimate, corrected exactly below)
  const float tn = 2.0f * nt + 1.0f;
  int ti = (int)((tn - sqrtf(fmaxf(tn * tn - 8.0f * t, 0.0f))) * 0.5f);
  auto row0 = [nt](int i) { return i * nt - i * (i - 1) / 2; };  // first triangle tile of tile row i
  while (ti > 0 && row0(ti) > t) --ti;
  while (ti + 1 < nt && row0(ti + 1) <= t) ++ti;
  *ti_ = ti;
  *tj_ = ti + (t - row0(ti));
}

// sum_{d1,d2} C1(d1) C2(d2) G(|D1 + d1|, |D2 + d2|) with C1 the correlation of
// k1 (K1 weights) and l1 (L1), C2 of k2 and l2
template <int K1, int L1, int K2, int L2>
__device__ __forceinline__ double term_sum(const double* k1, const double* l1, const double* k2, const double* l2,
                                           int D1, int D2, const double* __restrict__ G, int ld, int M) {
  double c1[K1 + L1 - 1], c2[K2 + L2 - 1];
#pragma unroll
  for (int d = 0; d < K1 + L1 - 1; ++d) c1[d] = 0.0;
#pragma unroll
  for (int d = 0; d < K2 + L2 - 1; ++d) c2[d] = 0.0;
#pragma unroll
  for (int t = 0; t < K1; ++t)
#pragma unroll
    for (int u = 0; u < L1; ++u) c1[t - u + L1 - 1] = fma(k1[t], l1[u], c1[t - u + L1 - 1]);
#pragma unroll
  for (int t = 0; t < K2; ++t)
#pragma unroll
    for (int u = 0; u < L2; ++u) c2[t - u + L2 - 1] = fma(k2[t], l2[u], c2[t - u + L2 - 1]);
  D1 -= L1 - 1;
  D2 -= L2 - 1;
  double acc = 0.0;
#pragma unroll
  for (int d1 = 0; d1 < K1 + L1 - 1; ++d1) {
    const double* row = G + (size_t)min(abs(D1 + d1), M) * ld;
    double part = 0.0;
#pragma unroll
    for (int d2 = 0; d2 < K2 + L2 - 1; ++d2) part = fma(c2[d2], __ldg(row + min(abs(D2 + d2), M)), part);
    acc = fma(c1[d1], part, acc);
  }
  return acc;
}

// A[k + N l] = sgn w_l T_kl, T_kl = sum_{p,q} c_kp c_lq sum_{dx,dy} Cx Cy G(...).
// T is symmetric (both sides have the same functionals): a CTA per 16 x 16 tile
// of its upper triangle writes both entries.  Bound by the FP64 rate: 88 FMAs
// per pair for plain interpolation, 450 with two terms.  All pairs with 5 x 5
// weights (140 and 560) took 148 us for 696 points, one term; this 46.
template <bool PLAIN>
__global__ void __launch_bounds__(256) k_schur_pairs(int N, int kind, const Functional* __restrict__ F,
                                                     const double* __restrict__ w, const double* __restrict__ G,
                                                     int ld, int M, double sgn, double* __restrict__ A) {
  int ti, tj;
  triangle_tile(blockIdx.x, (N + 15) / 16, &ti, &tj);
  const int k = ti * 16 + threadIdx.y, l = tj * 16 + threadIdx.x;
  if (k >= N || l >= N) return;
  const Functional& Fk = F[k];
  const Functional& Fl = F[l];
  double total = 0.0;
  if (PLAIN) {
    total = term_sum<NTAP, NTAP, NTAP, NTAP>(Fk.xw[0], Fl.xw[0], Fk.yw[0], Fl.yw[0], Fk.xb[0] - Fl.xb[0],
                                             Fk.yb[0] - Fl.yb[0], G, ld, M);
  } else {
#pragma unroll 1
    for (int p = 0; p < 2; ++p)
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const bool sx = short_in_x(kind, p);
        const double *k1 = sx ? Fk.xw[p] : Fk.yw[p], *k2 = sx ? Fk.yw[p] : Fk.xw[p];
        const double *l1 = sx ? Fl.xw[q] : Fl.yw[q], *l2 = sx ? Fl.yw[q] : Fl.xw[q];
        const int dx = Fk.xb[p] - Fl.xb[q], dy = Fk.yb[p] - Fl.yb[q];
        const int D1 = sx ? dx : dy, D2 = sx ? dy : dx;
        const double acc = p == q ? term_sum<NTAP, NTAP, FW, FW>(k1, l1, k2, l2, D1, D2, G, ld, M)
                                  : term_sum<NTAP, FW, FW, NTAP>(k1, l1, k2, l2, D1, D2, G, ld, M);
        total = fma(Fk.coef[p] * Fl.coef[q], acc, total);
      }
  }
  A[(size_t)l * N + k] = sgn * (w ? w[l] : 1.0) * total;
  if (ti != tj) A[(size_t)k * N + l] = sgn * (w ? w[k] : 1.0) * total;
}

// nRTRn: A[k + N l] = scale * w_l * (nx_k nx_l <phiU_k,phiU_l> + ny_k ny_l <phiV_k,phiV_l>)
__global__ void k_nrtrn(int N, const int* __restrict__ bxP, const int* __restrict__ bxD, const int* __restrict__ byP,
                        const int* __restrict__ byD, const double* __restrict__ wxP, const double* __restrict__ wxD,
                        const double* __restrict__ wyP, const double* __restrict__ wyD, const double* __restrict__ nx,
                        const double* __restrict__ ny, const double* __restrict__ w, double scale,
                        double* __restrict__ A) {
  const int k = blockIdx.y * 16 + threadIdx.y;
  const int l = blockIdx.x * 16 + threadIdx.x;
  if (k >= N || l >= N) return;
  auto ov = [&](const int* b, const double* wv) {
    const int d = b[k] - b[l];
    double s = 0.0;
    for (int t = 0; t < NTAP; ++t) {
      const int u = t + d;
      if (u >= 0 && u < NTAP) s += wv[(size_t)k * NTAP + t] * wv[(size_t)l * NTAP + u];
    }
    return s;
  };
  const double su = ov(bxD, wxD) * ov(byP, wyP);
  const double sv = ov(bxP, wxP) * ov(byD, wyD);
  A[(size_t)l * N + k] = scale * w[l] * (nx[k] * nx[l] * su + ny[k] * ny[l] * sv);
}

int schur_build(ilm_cache_s* c, int which, double scale, double* A, cudaStream_t st, bool any_cache) {
  const int N = c->npts;
  if (N == 0) return ILM_OK;
  const ilm_grid_s& g = c->grid;
  dim3 blk(16, 16), grd((N + 15) / 16, (N + 15) / 16);
  if (which == ILM_SCHUR_NRTRN) {
    // R_f = diag(ds/h^2) phi (GridScaling) or phi (IndexScaling); E = phi
    DevBuf W;
    ILM_TRY(W.alloc((size_t)N * sizeof(double)));
    if (c->scaling == ILM_GRID_SCALING) {
      ILM_TRY(st_axpby(N, ILM_F64, 1.0 / (g.h * g.h), c->ds64.p, 0.0, nullptr, W.p, st));
    } else {
      ILM_TRY(st_fill(N, ILM_F64, 1.0, W.p, st));
    }
    k_nrtrn<<<grd, blk, 0, st>>>(N, c->bx[0].as<int>(), c->bx[1].as<int>(), c->by[0].as<int>(), c->by[1].as<int>(),
                                 c->wx64[0].as<double>(), c->wx64[1].as<double>(), c->wy64[0].as<double>(),
                                 c->wy64[1].as<double>(), c->nx64.as<double>(), c->ny64.as<double>(),
                                 W.as<double>(), scale, A);
    ILM_CHECK_LAUNCH();
    ILM_CHECK_CUDA(cudaStreamSynchronize(st));
    return ILM_OK;
  }
  if (c->kind == ILM_CACHE_VECTOR && !any_cache) {
    set_error("dense Schur build for vector caches not supported");
    return ILM_ERR_UNSUPPORTED;
  }
  const double* G = nullptr;
  int ld = 0;
  const int M = std::max(g.nx, g.ny) + 16;
  ILM_TRY(lgf_table_device(M, &G, &ld, st));
  DevBuf& F = c->schur_F;
  if (F.bytes < (size_t)N * sizeof(Functional)) ILM_TRY(F.alloc((size_t)N * sizeof(Functional)));
  const double invh = c->scaling == ILM_GRID_SCALING ? 1.0 / g.h : 1.0;
  // w_l = regularization weight / factor : GridScaling ds_l/h^2 * h^2 = ds_l
  k_functionals<<<(N + 127) / 128, 128, 0, st>>>(N, which, c->bx[0].as<int>(), c->bx[1].as<int>(), c->by[0].as<int>(),
                                                 c->by[1].as<int>(), c->wx64[0].as<double>(), c->wx64[1].as<double>(),
                                                 c->wy64[0].as<double>(), c->wy64[1].as<double>(),
                                                 c->nx64.as<double>(), c->ny64.as<double>(), invh, F.as<Functional>());
  ILM_CHECK_LAUNCH();
  // RTLinvR: -scale ; CLinvCT: -scale ; GLinvD: +scale (G_s = -D_s^T)
  const double sgn = (which == ILM_SCHUR_GLINVD) ? scale : -scale;
  const double* w = c->scaling == ILM_GRID_SCALING ? c->ds64.as<double>() : nullptr;
  const int nt = (N + 15) / 16;
  (which == ILM_SCHUR_RTLINVR ? k_schur_pairs<true> : k_schur_pairs<false>)<<<nt * (nt + 1) / 2, blk, 0, st>>>(
      N, which, F.as<Functional>(), w, G, ld, ld - 1, sgn, A);
  ILM_CHECK_LAUNCH();
  return ILM_OK;
}

}  // namespace ilm

// ---------------------------------------------------------------------------
// batched Schur builds: all problems of a batch in one launch
// ---------------------------------------------------------------------------
namespace ilm {

__global__ void k_functionals_batched(int Ptot, const int* __restrict__ pt2prob, const SchurProbDev* __restrict__ pr,
                                      const int* __restrict__ bxP, const int* __restrict__ bxD,
                                      const int* __restrict__ byP, const int* __restrict__ byD,
                                      const double* __restrict__ wxP, const double* __restrict__ wxD,
                                      const double* __restrict__ wyP, const double* __restrict__ wyD,
                                      const double* __restrict__ nx, const double* __restrict__ ny,
                                      const double* __restrict__ w, Functional* __restrict__ out, int force_kind) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= Ptot) return;
  SchurProbDev P = pr[pt2prob[g]];
  if (force_kind >= 0) P.kind = force_kind;
  // reuse the single-problem kernel body on a one-point view
  const int k = g;
  Functional F;
  for (int p = 0; p < 2; ++p) {
    F.coef[p] = 0.0;
    F.xb[p] = F.yb[p] = 0;
    for (int t = 0; t < FW; ++t) F.xw[p][t] = F.yw[p][t] = 0.0;
  }
  const double* wxp = wxP + (size_t)k * NTAP;
  const double* wxd = wxD + (size_t)k * NTAP;
  const double* wyp = wyP + (size_t)k * NTAP;
  const double* wyd = wyD + (size_t)k * NTAP;
  auto at = [](const double* w, int t) { return (t >= 0 && t < NTAP) ? w[t] : 0.0; };
  if (P.kind == ILM_SCHUR_RTLINVR) {
    F.nterm = 1;
    F.coef[0] = 1.0;
    F.xb[0] = bxP[k];
    F.yb[0] = byP[k];
    for (int t = 0; t < NTAP; ++t) {
      F.xw[0][t] = wxp[t];
      F.yw[0][t] = wyp[t];
    }
  } else if (P.kind == ILM_SCHUR_GLINVD) {  // D_s functional on Nodes{Primal} (as k_functionals)
    F.nterm = 2;
    F.coef[0] = nx[k] * P.invh;
    F.xb[0] = bxD[k] - 1;
    F.yb[0] = byP[k];
    for (int t = 0; t < FW; ++t) {
      F.xw[0][t] = at(wxd, t) - at(wxd, t - 1);
      F.yw[0][t] = at(wyp, t);
    }
    F.coef[1] = ny[k] * P.invh;
    F.xb[1] = bxP[k];
    F.yb[1] = byD[k] - 1;
    for (int t = 0; t < FW; ++t) {
      F.xw[1][t] = at(wxp, t);
      F.yw[1][t] = at(wyd, t) - at(wyd, t - 1);
    }
  } else {  // CLinvCT
    F.nterm = 2;
    F.coef[0] = nx[k] * P.invh;
    F.xb[0] = bxD[k];
    F.yb[0] = byP[k];
    for (int t = 0; t < FW; ++t) {
      F.xw[0][t] = at(wxd, t);
      F.yw[0][t] = at(wyp, t - 1) - at(wyp, t);
    }
    F.coef[1] = ny[k] * P.invh;
    F.xb[1] = bxP[k];
    F.yb[1] = byD[k];
    for (int t = 0; t < FW; ++t) {
      F.xw[1][t] = at(wxp, t) - at(wxp, t - 1);
      F.yw[1][t] = at(wyd, t);
    }
  }
  FunctionalFF Q;
  Q.nterm = (short)F.nterm;
  Q.pad_[0] = Q.pad_[1] = Q.pad_[2] = 0;
  {
    const double wk = w ? w[g] : 0.0;
    const float wh = (float)wk;
    Q.w[0] = wh;
    Q.w[1] = (float)(wk - (double)wh);
  }
  for (int p = 0; p < 2; ++p) {
    Q.xb[p] = (short)F.xb[p];
    Q.yb[p] = (short)F.yb[p];
    const float ch = (float)F.coef[p];
    Q.coef[p][0] = ch;
    Q.coef[p][1] = (float)(F.coef[p] - (double)ch);
    for (int t = 0; t < FW; ++t) {
      const float xh = (float)F.xw[p][t], yh = (float)F.yw[p][t];
      Q.xw[p][t][0] = xh;
      Q.xw[p][t][1] = (float)(F.xw[p][t] - (double)xh);
      Q.yw[p][t][0] = yh;
      Q.yw[p][t][1] = (float)(F.yw[p][t] - (double)yh);
    }
  }
  reinterpret_cast<FunctionalFF*>(out)[g] = Q;
}


// Batched Schur entries in float-float on the FP32 pipes (~2^-44 relative
// per operation; GB300 issues FP64 at a small fraction of its FP32 rate):
// the same 1-D weight correlations and LGF contractions as k_schur_pairs,
// with the weights read as float-float pairs (split once per point) and the
// LGF read from its float-float copy.
//
// T_kl = sum_{p,q} c_p c_q sum_{dx,dy} Cx(dx) Cy(dy) G(|Dx + dx|, |Dy + dy|)
// for the functionals of points k and l (Cx, Cy the 1-D correlations of their
// weights).
__device__ __forceinline__ FF pair_sum(const FunctionalFF& Fk, const FunctionalFF& Fl, const float2* __restrict__ G,
                                       int ld, int M) {
  FF total{0.f, 0.f};
  for (int p = 0; p < Fk.nterm; ++p) {
    FF xk[FW], yk[FW];
#pragma unroll
    for (int a = 0; a < FW; ++a) {
      xk[a] = FF{Fk.xw[p][a][0], Fk.xw[p][a][1]};
      yk[a] = FF{Fk.yw[p][a][0], Fk.yw[p][a][1]};
    }
    for (int q = 0; q < Fl.nterm; ++q) {
      FF cx[2 * FW - 1], cy[2 * FW - 1];
#pragma unroll
      for (int d = 0; d < 2 * FW - 1; ++d) cx[d] = cy[d] = FF{0.f, 0.f};
#pragma unroll
      for (int b = 0; b < FW; ++b) {
        const float xbh = Fl.xw[q][b][0], xbl = Fl.xw[q][b][1];
        const float ybh = Fl.yw[q][b][0], ybl = Fl.yw[q][b][1];
#pragma unroll
        for (int a = 0; a < FW; ++a) {
          ff_fma(cx[a - b + FW - 1], xk[a].hi, xk[a].lo, xbh, xbl);
          ff_fma(cy[a - b + FW - 1], yk[a].hi, yk[a].lo, ybh, ybl);
        }
      }
#pragma unroll
      for (int d = 0; d < 2 * FW - 1; ++d) {
        cx[d] = ff_renorm(cx[d].hi, cx[d].lo);
        cy[d] = ff_renorm(cy[d].hi, cy[d].lo);
      }
      const int Dx = Fk.xb[p] - Fl.xb[q] - (FW - 1);
      const int Dy = Fk.yb[p] - Fl.yb[q] - (FW - 1);
      FF acc{0.f, 0.f};
#pragma unroll
      for (int dy = 0; dy < 2 * FW - 1; ++dy) {
        int my = abs(Dy + dy);
        my = my > M ? M : my;
        const float2* Grow = G + (size_t)my;
        FF racc{0.f, 0.f};
#pragma unroll
        for (int dx = 0; dx < 2 * FW - 1; ++dx) {
          int mx = abs(Dx + dx);
          mx = mx > M ? M : mx;
          const float2 g = __ldg(Grow + (size_t)mx * ld);
          ff_fma(racc, g.x, g.y, cx[dx].hi, cx[dx].lo);
        }
        racc = ff_renorm(racc.hi, racc.lo);
        ff_fma(acc, cy[dy].hi, cy[dy].lo, racc.hi, racc.lo);
      }
      acc = ff_renorm(acc.hi, acc.lo);
      const FF cc = ff_mul(FF{Fk.coef[p][0], Fk.coef[p][1]}, FF{Fl.coef[q][0], Fl.coef[q][1]});
      ff_fma(total, cc.hi, cc.lo, acc.hi, acc.lo);
    }
  }
  return ff_renorm(total.hi, total.lo);
}

// The LGF as the pairs of one tile read it: the patch of distances that the
// tile needs in shared memory where it fits (a few thousand entries for points
// that follow a curve), else the table.  Read from the table by every pair,
// the gathers took two thirds of the load / store pipe; with the patch, the
// short axes' four weights and a rolled loop (the unrolled one waited for its
// instructions) the two-term tiles of 64 problems go from 386
// to 300 us, bound by the float-float issue rate.
constexpr int PATCH = 5888;  // entries (46 KB: three CTAs per SM)
constexpr int FFN = sizeof(FunctionalFF) / 4, FFW = (FFN + 3) / 4 * 4 + 2;  // words of a functional, and its stride
static_assert(sizeof(FunctionalFF) % 4 == 0 && (FFW / 2) % 2 == 1, "16 functionals' pairs lie in distinct banks");
constexpr size_t PAIR_SMEM = 32 * FFW * sizeof(float) + (PATCH + 256 * (2 * FW - 1)) * sizeof(float2);

struct GPatch {
  const float2* G;
  int ld, M;
  const float2* patch;
  int ldp, x0, y0;
};

// as term_sum, in float-float; the first axis is x (XF) or y
template <bool SMEM, int K1, int L1, int K2, int L2>
__device__ __forceinline__ FF term_sum_ff(const float (*k1)[2], const float (*l1)[2], const float (*k2)[2],
                                          const float (*l2)[2], int D1, int D2, bool xf, const GPatch& g,
                                          float2* col) {
  FF c1[K1 + L1 - 1], c2[K2 + L2 - 1];
#pragma unroll
  for (int d = 0; d < K1 + L1 - 1; ++d) c1[d] = FF{0.f, 0.f};
#pragma unroll
  for (int d = 0; d < K2 + L2 - 1; ++d) c2[d] = FF{0.f, 0.f};
#pragma unroll
  for (int u = 0; u < L1; ++u) {
    const float2 b = *reinterpret_cast<const float2*>(l1[u]);
#pragma unroll
    for (int t = 0; t < K1; ++t) ff_fma(c1[t - u + L1 - 1], k1[t][0], k1[t][1], b.x, b.y);
  }
#pragma unroll
  for (int u = 0; u < L2; ++u) {
    const float2 b = *reinterpret_cast<const float2*>(l2[u]);
#pragma unroll
    for (int t = 0; t < K2; ++t) ff_fma(c2[t - u + L2 - 1], k2[t][0], k2[t][1], b.x, b.y);
  }
#pragma unroll
  for (int d = 0; d < K1 + L1 - 1; ++d) {
    c1[d] = ff_renorm(c1[d].hi, c1[d].lo);
    col[d * 256] = make_float2(c1[d].hi, c1[d].lo);
  }
#pragma unroll
  for (int d = 0; d < K2 + L2 - 1; ++d) c2[d] = ff_renorm(c2[d].hi, c2[d].lo);
  D1 -= L1 - 1;
  D2 -= L2 - 1;
  const int st1 = SMEM ? (xf ? g.ldp : 1) : (xf ? g.ld : 1), st2 = SMEM ? (xf ? 1 : g.ldp) : (xf ? 1 : g.ld);
  const int o1 = SMEM ? (xf ? g.x0 : g.y0) : 0, o2 = SMEM ? (xf ? g.y0 : g.x0) : 0;
  int at2[K2 + L2 - 1];
#pragma unroll
  for (int d = 0; d < K2 + L2 - 1; ++d) {
    const int m = abs(D2 + d);
    at2[d] = ((SMEM ? m : min(m, g.M)) - o2) * st2;
  }
  FF acc{0.f, 0.f};
#pragma unroll 1
  for (int d1 = 0; d1 < K1 + L1 - 1; ++d1) {
    const int m = abs(D1 + d1);
    const float2 w1 = col[d1 * 256];
    const float2* row = (SMEM ? g.patch : g.G) + ((SMEM ? m : min(m, g.M)) - o1) * st1;
    FF part{0.f, 0.f};
#pragma unroll
    for (int d2 = 0; d2 < K2 + L2 - 1; ++d2) {
      const float2 v = SMEM ? row[at2[d2]] : __ldg(row + at2[d2]);
      ff_fma(part, v.x, v.y, c2[d2].hi, c2[d2].lo);
    }
    part = ff_renorm(part.hi, part.lo);
    ff_fma(acc, w1.x, w1.y, part.hi, part.lo);
  }
  return ff_renorm(acc.hi, acc.lo);
}

// T_kl of one problem's kind
template <bool SMEM>
__device__ __forceinline__ FF schur_pair(int kind, const FunctionalFF& Fk, const FunctionalFF& Fl, const GPatch& g,
                                         float2* col) {
  if (kind == ILM_SCHUR_RTLINVR)
    return term_sum_ff<SMEM, NTAP, NTAP, NTAP, NTAP>(Fk.xw[0], Fl.xw[0], Fk.yw[0], Fl.yw[0], Fk.xb[0] - Fl.xb[0],
                                                     Fk.yb[0] - Fl.yb[0], true, g, col);
  FF total{0.f, 0.f};
#pragma unroll 1
  for (int p = 0; p < 2; ++p)
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      const bool sx = short_in_x(kind, p);
      const float(*k1)[2] = sx ? Fk.xw[p] : Fk.yw[p];
      const float(*k2)[2] = sx ? Fk.yw[p] : Fk.xw[p];
      const float(*l1)[2] = sx ? Fl.xw[q] : Fl.yw[q];
      const float(*l2)[2] = sx ? Fl.yw[q] : Fl.xw[q];
      const int dx = Fk.xb[p] - Fl.xb[q], dy = Fk.yb[p] - Fl.yb[q];
      const int D1 = sx ? dx : dy, D2 = sx ? dy : dx;
      const FF acc = p == q ? term_sum_ff<SMEM, NTAP, NTAP, FW, FW>(k1, l1, k2, l2, D1, D2, sx, g, col)
                            : term_sum_ff<SMEM, NTAP, FW, FW, NTAP>(k1, l1, k2, l2, D1, D2, sx, g, col);
      const FF cc = ff_mul(FF{Fk.coef[p][0], Fk.coef[p][1]}, FF{Fl.coef[q][0], Fl.coef[q][1]});
      ff_fma(total, cc.hi, cc.lo, acc.hi, acc.lo);
    }
  return ff_renorm(total.hi, total.lo);
}

__global__ void __launch_bounds__(256) k_schur_pairs_batched(int nprob, const SchurProbDev* __restrict__ pr,
                                                             const FunctionalFF* __restrict__ F,
                                                             const double* __restrict__ w,
                                                             const float2* __restrict__ G, int ld, int M,
                                                             float* __restrict__ Shi, float* __restrict__ Slo) {
  int lo = 0, hi = nprob - 1;
  const int u = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pr[mid].tile0 <= u) lo = mid; else hi = mid - 1;
  }
  const SchurProbDev P = pr[lo];
  const int N = P.n;
  const int nt = (N + 15) / 16;
  // the tile sum T_kl = sum U_k(a) G(a - b) U_l(b) is symmetric (G depends on
  // |a - b| only and both sides use the same functionals): one CTA per tile
  // of the upper triangle (ti <= tj) in row-major order, writing S_kl = -w_l
  // T_kl and, off the diagonal tiles, S_lk = -w_k T_kl
  int ti, tj;
  triangle_tile(u - P.tile0, nt, &ti, &tj);
  const int k = ti * 16 + threadIdx.y;
  const int l = tj * 16 + threadIdx.x;
  extern __shared__ __align__(16) unsigned char smraw[];
  float* sf = reinterpret_cast<float*>(smraw);  // functionals of the tile's 16 + 16 points
  float2* patch = reinterpret_cast<float2*>(sf + 32 * FFW);
  float2* col = patch + PATCH + threadIdx.y * 16 + threadIdx.x;  // the thread's first correlation (the loop over it is rolled)
  __shared__ int s_lo[4], s_hi[4];  // x and y bases of the k points, then of the l points
  {
    const int tid = threadIdx.y * 16 + threadIdx.x;
    if (tid < 4) {
      s_lo[tid] = 0x7fffffff;
      s_hi[tid] = -0x7fffffff;
    }
    for (int e = tid; e < 32 * FFN; e += 256) {
      const int i = e / FFN, f = e - i * FFN, g = i < 16 ? ti * 16 + i : tj * 16 + i - 16;
      if (g < N) sf[i * FFW + f] = reinterpret_cast<const float*>(F + P.poff + g)[f];
    }
    __syncthreads();
    if (tid < 64) {  // (point, term)
      const int i = tid >> 1, q = tid & 1, g = i < 16 ? ti * 16 + i : tj * 16 + i - 16;
      const FunctionalFF& f = *reinterpret_cast<const FunctionalFF*>(sf + i * FFW);
      if (g < N && q < f.nterm) {
        const int s = i < 16 ? 0 : 2;
        atomicMin(&s_lo[s], (int)f.xb[q]);
        atomicMax(&s_hi[s], (int)f.xb[q]);
        atomicMin(&s_lo[s + 1], (int)f.yb[q]);
        atomicMax(&s_hi[s + 1], (int)f.yb[q]);
      }
    }
    __syncthreads();
  }
  // distances of the tile: [lo, hi] per axis, FW - 1 beyond the bases' on both sides
  GPatch gp{G, ld, M, nullptr, 0, 0, 0};
  {
    int lo[2], hi[2];
    for (int a = 0; a < 2; ++a) {
      const int d0 = s_lo[a] - s_hi[2 + a] - (FW - 1), d1 = s_hi[a] - s_lo[2 + a] + (FW - 1);
      lo[a] = d0 <= 0 && d1 >= 0 ? 0 : min(abs(d0), abs(d1));
      hi[a] = max(abs(d0), abs(d1));
    }
    // (an odd row stride: the lanes' points lie along a curve)
    const int nx = hi[0] - lo[0] + 1, ny = hi[1] - lo[1] + 1, ldp = ny | 1;
    if ((long long)nx * ldp <= PATCH && hi[0] <= M && hi[1] <= M) {
      for (int e = threadIdx.y * 16 + threadIdx.x; e < nx * ny; e += 256) {
        const int i = e / ny, j = e - i * ny;
        patch[i * ldp + j] = __ldg(G + (size_t)(lo[0] + i) * ld + lo[1] + j);
      }
      gp.patch = patch;
      gp.ldp = ldp;
      gp.x0 = lo[0];
      gp.y0 = lo[1];
    }
    __syncthreads();
  }
  if (k >= N || l >= N) return;
  const FunctionalFF& Fk = *reinterpret_cast<const FunctionalFF*>(sf + threadIdx.y * FFW);
  const FunctionalFF& Fl = *reinterpret_cast<const FunctionalFF*>(sf + (16 + threadIdx.x) * FFW);
  const FF total = gp.patch ? schur_pair<true>(P.kind, Fk, Fl, gp, col) : schur_pair<false>(P.kind, Fk, Fl, gp, col);
  // row-major float-float pair: S[k][l] = hi + lo
  const FF wl{-Fl.w[0], -Fl.w[1]};
  const FF v = ff_mul(wl, total);
  Shi[P.soff + (size_t)k * schur_ld(N) + l] = v.hi;
  Slo[P.soff + (size_t)k * schur_ld(N) + l] = v.lo;
  if (ti != tj) {
    const FF wk{-Fk.w[0], -Fk.w[1]};
    const FF vt = ff_mul(wk, total);
    Shi[P.soff + (size_t)l * schur_ld(N) + k] = vt.hi;
    Slo[P.soff + (size_t)l * schur_ld(N) + k] = vt.lo;
  }
}

int schur_build_batched(int nprob, const SchurProbDev* probs_dev, int total_tiles, int Ptot, const int* pt2prob,
                        const BatchWin& W, const double* w, Functional* F, float* Shi, float* Slo, int max_grid,
                        cudaStream_t st, const SchurProbDev* order, int nfirst, int tiles_first,
                        cudaEvent_t mid) {
  if (Ptot == 0) return ILM_OK;
  const float2* G = nullptr;
  int ld = 0;
  ILM_TRY(lgf_table_ff_device(max_grid + 16, &G, &ld, st));
  k_functionals_batched<<<(Ptot + 127) / 128, 128, 0, st>>>(Ptot, pt2prob, probs_dev, W.bx[0], W.bx[1], W.by[0],
                                                            W.by[1], W.wx64[0], W.wx64[1], W.wy64[0], W.wy64[1],
                                                            W.nx64, W.ny64, w, F, -1);
  ILM_CHECK_LAUNCH();
  // the pair tiles: one launch over probs_dev, or two over the build order
  // (the functionals above index probs_dev by problem, so it stays in
  // problem order)
  const FunctionalFF* FF_ = reinterpret_cast<const FunctionalFF*>(F);
  ILM_CHECK_CUDA(cudaFuncSetAttribute(k_schur_pairs_batched, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PAIR_SMEM));
  if (!order) {
    if (total_tiles > 0)
      k_schur_pairs_batched<<<total_tiles, dim3(16, 16), PAIR_SMEM, st>>>(nprob, probs_dev, FF_, w, G, ld, ld - 1, Shi, Slo);
    ILM_CHECK_LAUNCH();
    return ILM_OK;
  }
  if (tiles_first > 0)
    k_schur_pairs_batched<<<tiles_first, dim3(16, 16), PAIR_SMEM, st>>>(nfirst, order, FF_, w, G, ld, ld - 1, Shi, Slo);
  ILM_CHECK_LAUNCH();
  if (mid) ILM_CHECK_CUDA(cudaEventRecord(mid, st));
  const int tiles_second = total_tiles - tiles_first;
  if (tiles_second > 0)
    k_schur_pairs_batched<<<tiles_second, dim3(16, 16), PAIR_SMEM, st>>>(nprob - nfirst, order + nfirst, FF_, w, G, ld,
                                                                 ld - 1, Shi, Slo);
  ILM_CHECK_LAUNCH();
  return ILM_OK;
}

// The right-hand-side operator of the batched solves, built from the same
// LGF point-point sums as S: Dirichlet M = E L^-1 D_s (the Schur right-hand
// side E f*, f* = L^-1 D_s [f]), Neumann M = G_s L^-1 R (G_s f*, f* =
// L^-1 R [v_n]).  With the plain-interpolation functionals U and the double-
// layer functionals D of k_functionals, E L^-1 R = w_l U G U and
// G_s = -D^T, so M_kl = +w_l (U G D)_kl (Dirichlet) and -w_l (D G U)_kl
// (Neumann).  Full n x n tiles (M is not symmetric), one CTA per 16 x 16
// tile, float-float as k_schur_pairs_batched; the tiles of problem p start at
// pr[p].tile0 (the caller's full-tile numbering).
__global__ void __launch_bounds__(256) k_rhsop_pairs_batched(int nprob, const SchurProbDev* __restrict__ pr,
                                                             const FunctionalFF* __restrict__ FU,
                                                             const FunctionalFF* __restrict__ FD,
                                                             const double* __restrict__ w,
                                                             const float2* __restrict__ G, int ld, int M,
                                                             float* __restrict__ Mhi, float* __restrict__ Mlo) {
  int lo = 0, hi = nprob - 1;
  const int u = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pr[mid].tile0 <= u) lo = mid; else hi = mid - 1;
  }
  const SchurProbDev P = pr[lo];
  const int N = P.n;
  const int nt = (N + 15) / 16;
  const int t = u - P.tile0;
  const int ti = t / nt, tj = t - (t / nt) * nt;
  const int k = ti * 16 + threadIdx.y;
  const int l = tj * 16 + threadIdx.x;
  if (k >= N || l >= N) return;
  const bool dir = P.kind == ILM_SCHUR_RTLINVR;
  const FunctionalFF& Fl = dir ? FD[P.poff + l] : FU[P.poff + l];
  const FF total = pair_sum(dir ? FU[P.poff + k] : FD[P.poff + k], Fl, G, ld, M);
  const FF wl = dir ? FF{Fl.w[0], Fl.w[1]} : FF{-Fl.w[0], -Fl.w[1]};
  const FF v = ff_mul(wl, total);
  Mhi[P.soff + (size_t)k * schur_ld(N) + l] = v.hi;
  Mlo[P.soff + (size_t)k * schur_ld(N) + l] = v.lo;
}

int rhsop_build_batched(int nprob, const SchurProbDev* probs_full_dev, int total_tiles, int Ptot, const int* pt2prob,
                        const BatchWin& W, const double* w, Functional* FU, Functional* FD, float* Mhi, float* Mlo,
                        int max_grid, cudaStream_t st) {
  if (Ptot == 0) return ILM_OK;
  const float2* G = nullptr;
  int ld = 0;
  ILM_TRY(lgf_table_ff_device(max_grid + 16, &G, &ld, st));
  k_functionals_batched<<<(Ptot + 127) / 128, 128, 0, st>>>(Ptot, pt2prob, probs_full_dev, W.bx[0], W.bx[1], W.by[0],
                                                            W.by[1], W.wx64[0], W.wx64[1], W.wy64[0], W.wy64[1],
                                                            W.nx64, W.ny64, w, FU, ILM_SCHUR_RTLINVR);
  ILM_CHECK_LAUNCH();
  k_functionals_batched<<<(Ptot + 127) / 128, 128, 0, st>>>(Ptot, pt2prob, probs_full_dev, W.bx[0], W.bx[1], W.by[0],
                                                            W.by[1], W.wx64[0], W.wx64[1], W.wy64[0], W.wy64[1],
                                                            W.nx64, W.ny64, w, FD, ILM_SCHUR_GLINVD);
  ILM_CHECK_LAUNCH();
  k_rhsop_pairs_batched<<<total_tiles, dim3(16, 16), 0, st>>>(nprob, probs_full_dev,
                                                              reinterpret_cast<const FunctionalFF*>(FU),
                                                              reinterpret_cast<const FunctionalFF*>(FD), w, G, ld,
                                                              ld - 1, Mhi, Mlo);
  ILM_CHECK_LAUNCH();
  return ILM_OK;
}

size_t functional_size() { return sizeof(Functional); }

}  // namespace ilm
