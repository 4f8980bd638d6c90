// FP64 CG of one problem: the Schur solves of single caches (dense S) and the
// stage systems of the heat march (sparse S).
//
// GB300 issues two FP64 FMAs per clock and SM, so a product with a dense
// n x n matrix costs n^2 / 2 clocks on one SM (n = 448: 50 us) and has to be
// spread over many of them; what is left of an iteration is latency -- the
// exchange between CTAs, block reductions, the CG scalars.  Each CTA
// therefore owns a slice of the rows of S, kept in shared memory for the
// whole solve where it fits, and holds every vector of the recurrence in
// full: a product's rows are sent to all CTAs, one barrier publishes them,
// and every CTA runs the same vector updates and reductions on the same
// numbers in the same order.  One barrier per iteration, bit-identical
// scalars everywhere, so all CTAs take the same branches.
//
// Before the iteration, an FP32 inverse of W S (formed once per S) is refined
// with FP64 residuals: x += P (b - S x).  Each step gains cond(S) eps_32, so a
// few steps, each one product with S and one (cheap) with P, replace the ~60
// to ~300 iterations; the residual that is tested is the FP64 one.  Where a
// step gains less than a factor of four the CG goes on from there.
//
// Two exchanges: a single cluster of 16 CTAs (rows written straight into the
// other CTAs' shared memory, hardware cluster barrier), and a cooperative
// grid of one CTA per SM (rows through L2, counter barrier with a bounded
// wait) for the larger problems, where the product of 16 SMs costs more than
// the slower barrier.
//
// Measured, us per iteration: n = 157 4.8, 448 7.1, 696 8.0, 1200 11.5, 2500
// 27.9 (one CTA per problem, the matrix streamed through one SM: about 24, 62
// and 167 at n = 157, 448, 696).  Up to n ~ 700 the iteration is a chain of dependent
// FP64 operations (64 clocks each: two block reductions, two divides), above
// it the FP64 issue rate of the product.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include "ilm_internal.cuh"

namespace cg = cooperative_groups;

namespace ilm {
namespace {

constexpr int C64_T = 256;             // threads per CTA
constexpr int C64_CLUSTER = 16;        // CTAs of the cluster variant
constexpr int C64_MAX_SMEM = 227 * 1024 - 256;  // dynamic shared memory beside the static scalars
// matrix entries up to which the cluster variant is used: an iteration of a
// dense n takes 4.8 / 5.4 / 6.9 / 8.2 us with the cluster and 5.5 / 5.8 / 6.8 /
// 6.9 us with the grid at n = 157 / 224 / 300 / 400
constexpr long long C64_CLUSTER_ENTRIES = 256 * 256;
constexpr unsigned C64_SPIN = 1u << 22;  // polls of the grid barrier before it gives up (seconds)

struct CG64Args {
  CG64Problem p;
  int R;            // rows per CTA
  int lpr;          // lanes per row of the product (4, 8, 16, 32)
  int resident;     // the CTA's rows of S are kept in shared memory
  int ld;           // row stride of the resident dense slab (doubles)
  int slab_nnz;     // CSR: entries of the largest slab
  double* gq;       // grid variant: two exchange buffers of n doubles
  CG64State* state;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// shared-memory scalars: [0, 8) and [8, 16) warp partials, then the results
struct Scal {
  double part[16];
  float part32[8];
  double a, b, c;   // first sum, second sum, derived scalar
  int flag;
};

// Sums of a and b over the CTA (fixed order); thread 0 then derives
// s.c = fin(sum a, sum b).  Threads past the vectors' length hold zeros and
// their warps skip the shuffles.
template <typename F>
__device__ __forceinline__ void block_sums(double a, double b, bool two, int n, Scal& s, F fin) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp * 32 < n) {
    a = warp_sum(a);
    if (two) b = warp_sum(b);
  }
  if (lane == 0) {
    s.part[warp] = a;
    s.part[8 + warp] = b;
  }
  __syncthreads();
  if (warp == 0) {
    double u = lane < 16 ? s.part[lane] : 0.0;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) u += __shfl_xor_sync(0xffffffffu, u, o);
    const double v = __shfl_sync(0xffffffffu, u, 8);
    if (lane == 0) {
      s.a = u;
      s.b = v;
      fin(u, v);
    }
  }
  __syncthreads();
}

template <bool CSR, bool GRID>
__global__ void __launch_bounds__(C64_T, 1) k_cg64(const CG64Args A) {
  const CG64Problem& P = A.p;
  const int n = P.n, G = gridDim.x, rank = blockIdx.x, t = threadIdx.x;
  const int r0 = min(n, rank * A.R), nr = min(A.R, n - r0);
  extern __shared__ __align__(16) double sm[];
  double* x = sm;
  double* r = x + n;
  double* p = r + n;
  double* w = p + n;
  double* qb = w + n;                          // cluster: two buffers; grid: one
  double* slab = qb + (GRID ? 1 : 2) * (size_t)n;
  int* scol = reinterpret_cast<int*>(slab + A.slab_nnz);
  __shared__ Scal s;
  __shared__ int s_ok;
  int par = 0;           // exchange buffer
  unsigned bar = 0;      // grid barriers passed
  bool ok = true;

  int e0 = 0;
  if (CSR) e0 = P.rowptr[r0];
  if (A.resident) {
    if (CSR) {
      const int e1 = P.rowptr[r0 + nr];
      for (int e = e0 + t; e < e1; e += C64_T) {
        slab[e - e0] = (double)P.vhi[e] + (double)P.vlo[e];
        scol[e - e0] = P.colidx[e];
      }
    } else {
      for (int k = t; k < nr * n; k += C64_T) {
        const int j = k / nr, i = k - j * nr;
        slab[(size_t)i * A.ld + j] = P.A[(size_t)j * n + r0 + i];
      }
    }
  }

  // the CTAs' rows of one vector become visible to all
  auto publish = [&](double* q) {
    if (GRID) {
      // counter barrier: every CTA of the cooperative launch is resident; the
      // wait is bounded all the same
      __syncthreads();
      ++bar;
      if (t == 0) {
        __threadfence();
        atomicAdd(&A.state->arrived, 1u);
        const unsigned goal = bar * (unsigned)G;
        unsigned seen = 0, k = 0;
        do {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&A.state->arrived) : "memory");
        } while (seen < goal && ++k < C64_SPIN);
        s_ok = seen >= goal;
        if (seen < goal) atomicExch(P.timeout, 1);
      }
      __syncthreads();
      ok = s_ok != 0;
      for (int j = t; j < n; j += C64_T) q[j] = __ldcg(A.gq + (size_t)par * n + j);
      // no CTA barrier here: each thread reads back the entries it stored
    } else {
      cg::this_cluster().sync();
    }
    par ^= 1;
  };

  // rows r0 .. r0 + nr of P v for the FP32 inverse (v in shared memory, FP32),
  // each row a warp's, sent to every CTA
  auto product32 = [&](const float* v, float shift) -> double* {
    double* q = GRID ? qb : qb + (size_t)par * n;
    const int lane = t & 31, warp = t >> 5;
    for (int i = warp; i < nr; i += C64_T / 32) {
      const float* row = P.inv + (size_t)(r0 + i) * P.ldi;
      float a[4] = {0.f, 0.f, 0.f, 0.f};
      int j = lane;
      for (; j + 7 * 32 < n; j += 8 * 32) {  // eight loads from L2 in flight
        float m[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) m[q] = __ldg(row + j + 32 * q);
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q & 3] = fmaf(m[q], v[j + 32 * q], a[q & 3]);
      }
      {
        float m[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) m[q] = j + 32 * q < n ? __ldg(row + j + 32 * q) : 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (j + 32 * q < n) a[q & 3] = fmaf(m[q], v[j + 32 * q], a[q & 3]);
      }
      float a0 = (a[0] + a[1]) + (a[2] + a[3]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
      const double u = (double)fmaf(shift, __ldg(row + P.ldi - 32), a0);
      if (GRID) {
        if (lane == 0) __stcg(A.gq + (size_t)par * n + r0 + i, u);
      } else if (lane < G) {
        cg::this_cluster().map_shared_rank(q, lane)[r0 + i] = u;
      }
    }
    publish(q);
    return q;
  };

  // rows r0 .. r0 + nr of S v, sent to every CTA; returns the whole product
  // (cluster: the buffer the other CTAs wrote; grid: the CTA's own copy)
  auto product = [&](const double* v) -> double* {
    const int L = A.lpr, c = t & (L - 1), rows = C64_T / L;
    double* q = GRID ? qb : qb + (size_t)par * n;
    if (!CSR && GRID && !A.resident) {
      // S streamed from L2: consecutive threads take consecutive rows of one
      // column, partial sums meet in q (free between products; n > C64_T here)
      for (int b0 = 0; b0 < nr; b0 += C64_T) {
        const int m = min(C64_T, nr - b0), nc = C64_T / m, k = t / m, i = t - k * m;
        if (k < nc) {
          double a0 = 0.0, a1 = 0.0;
          const double* col = P.A + r0 + b0 + i;
          int j = k;
          for (; j + 3 * nc < n; j += 4 * nc) {
            const double s0 = __ldg(col + (size_t)j * n), s1 = __ldg(col + (size_t)(j + nc) * n);
            const double s2 = __ldg(col + (size_t)(j + 2 * nc) * n), s3 = __ldg(col + (size_t)(j + 3 * nc) * n);
            a0 = fma(s0, v[j], a0);
            a1 = fma(s1, v[j + nc], a1);
            a0 = fma(s2, v[j + 2 * nc], a0);
            a1 = fma(s3, v[j + 3 * nc], a1);
          }
          for (; j < n; j += nc) a0 = fma(__ldg(col + (size_t)j * n), v[j], a0);
          q[t] = a0 + a1;
        }
        __syncthreads();
        if (t < m) {
          double a = q[t];
          for (int u = 1; u < nc; ++u) a += q[u * m + t];
          __stcg(A.gq + (size_t)par * n + r0 + b0 + t, a);
        }
        __syncthreads();
      }
    } else {
      for (int i0 = 0; i0 < nr; i0 += rows) {
        const int i = i0 + t / L;
        double a0 = 0.0, a1 = 0.0;
        if (i < nr) {
          if (CSR) {
            const int b = P.rowptr[r0 + i], e = P.rowptr[r0 + i + 1];
            if (A.resident)
              for (int k = b + c; k < e; k += L) a0 = fma(slab[k - e0], v[scol[k - e0]], a0);
            else
              for (int k = b + c; k < e; k += L)
                a0 = fma((double)__ldg(P.vhi + k) + (double)__ldg(P.vlo + k), v[__ldg(P.colidx + k)], a0);
          } else {
            const double* row = slab + (size_t)i * A.ld;
            int j = c;
            for (; j + L < n; j += 2 * L) {
              a0 = fma(row[j], v[j], a0);
              a1 = fma(row[j + L], v[j + L], a1);
            }
            if (j < n) a0 = fma(row[j], v[j], a0);
          }
        }
        a0 += a1;
        for (int o = L >> 1; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        if (i < nr) {
          if (GRID) {
            if (c == 0) __stcg(A.gq + (size_t)par * n + r0 + i, a0);
          } else {
            cg::cluster_group cl = cg::this_cluster();
            for (int d = c; d < G; d += L) cl.map_shared_rank(q, d)[r0 + i] = a0;
          }
        }
      }
    }
    publish(q);
    return q;
  };

  for (int j = t; j < n; j += C64_T) {
    x[j] = P.x0 ? P.x0[j] : 0.0;
    w[j] = P.w ? P.w[j] : 1.0;
  }
  if (!GRID) cg::this_cluster().sync();  // every CTA of the cluster runs before its shared memory is written
  __syncthreads();
  if (P.x0) {  // warm start: r = b - S x0 (x0 may be the output: all CTAs have read it at the barrier)
    const double* q = product(x);
    for (int j = t; j < n; j += C64_T) r[j] = P.b[j] - q[j];
  } else {
    for (int j = t; j < n; j += C64_T) r[j] = P.b[j];
  }
  double bb = 0.0, rr = 0.0;
  for (int j = t; j < n; j += C64_T) {
    bb += P.b[j] * P.b[j];
    rr += r[j] * r[j];
  }
  block_sums(bb, rr, true, n, s, [](double, double) {});
  bb = s.a;
  rr = s.b;
  const double bnorm = sqrt(bb), thr = P.tol * bnorm, thr2 = thr * thr;
  // squared norms are compared, except where they are about to underflow
  auto below = [&](double v) { return v <= thr2 || v < 1e-280; };
  auto converged = [&](double v) { return thr2 > 1e-280 ? v <= thr2 : sqrt(v) <= thr; };
  int it = 0;
  bool done = bnorm == 0.0;
  double last = bb;
  if (P.inv && P.invs[0] != 0.f && !done) {
    float* v = reinterpret_cast<float*>(p);  // W r scaled into FP32's range
    const float kappa = P.invs[1];
    // x += P r, r the residual of squared norm rho
    auto correct = [&](double rho) {
      const int e = (__double2hiint(rho) >> 20 & 0x7ff) - 1023;  // rho ~ 2^e
      const double down = __hiloint2double((1023 - e / 2) << 20, 0), up = __hiloint2double((1023 + e / 2) << 20, 0);
      float g = 0.f, shift = 0.f;
      for (int j = t; j < n; j += C64_T) {
        const float vj = (float)(w[j] * (r[j] * down));
        v[j] = vj;
        if (kappa != 0.f) g = fmaf(__ldg(P.inv + (size_t)j * P.ldi + P.ldi - 32), vj, g);
      }
      if (kappa != 0.f) {
        for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
        if ((t & 31) == 0) s.part32[t >> 5] = g;
        __syncthreads();
        for (int k = 0; k < C64_T / 32; ++k) shift += s.part32[k];
        shift *= kappa;
      }
      __syncthreads();
      const double* u = product32(v, shift);
      for (int j = t; j < n; j += C64_T) x[j] = fma(u[j], up, x[j]);
      __syncthreads();
    };
    last = rr;
    done = converged(rr);
    bool slow = false;
    while (!done && !slow && ok && it < P.maxiter) {
      correct(last);
      if (!ok) break;
      const double* y = product(x);
      if (!ok) break;
      double tr = 0.0;
      for (int j = t; j < n; j += C64_T) {
        const double rj = P.b[j] - y[j];
        r[j] = rj;
        tr = fma(rj, rj, tr);
      }
      block_sums(tr, 0.0, false, n, s, [](double, double) {});
      ++it;
      const double now = s.a;
      done = converged(now);
      slow = !(now <= 0.0625 * last);
      if (slow && !done && !(now <= rr)) {  // no better than the start: the CG begins there
        for (int j = t; j < n; j += C64_T) x[j] = P.x0 ? P.x0[j] : 0.0;
        __syncthreads();
        if (P.x0) y = product(x);
        for (int j = t; j < n; j += C64_T) r[j] = P.x0 ? P.b[j] - y[j] : P.b[j];
        last = rr;
      } else {
        last = now;
      }
    }
    // The residual that passed is rich in the modes that P gets least right, the
    // slow ones, and x is further off for it than a CG iterate of that residual:
    // one correction more (its residual is not formed; steps gained a factor
    // of four so far)
    if (done && !slow && last > 0.0) correct(last);
  }
  double rz = 0.0;
  if (!done) {
    for (int j = t; j < n; j += C64_T) {
      p[j] = r[j];
      rz += w[j] * r[j] * r[j];
    }
    block_sums(rz, 0.0, false, n, s, [](double, double) {});
    rz = s.a;
  }
  const bool guard = P.stall > 0;
  double best = 1e300;
  int stalled = 0;
  if (guard)  // the best true-residual iterate is kept in P.x (each CTA its rows)
    for (int i = t; i < nr; i += C64_T) P.x[r0 + i] = x[r0 + i];
  __syncthreads();
  while (!done && ok && it < P.maxiter) {
    const double* q = product(p);
    if (!ok) break;
    double pq = 0.0;
    for (int j = t; j < n; j += C64_T) pq = fma(w[j] * p[j], q[j], pq);
    block_sums(pq, 0.0, false, n, s, [&](double u, double) { s.c = rz / u; });
    if (s.a == 0.0) break;
    const double alpha = s.c;
    double rs = 0.0, rzn = 0.0;
    for (int j = t; j < n; j += C64_T) {
      x[j] = fma(alpha, p[j], x[j]);
      const double rj = fma(-alpha, q[j], r[j]);
      r[j] = rj;
      const double r2 = rj * rj;
      rs += r2;
      rzn = fma(w[j], r2, rzn);
    }
    ++it;
    block_sums(rs, rzn, true, n, s, [&](double u, double v) {
      s.c = v / rz;
      s.flag = below(u);
    });
    last = s.a;
    rzn = s.b;
    double beta = s.c;
    if (s.flag || it % P.refresh == 0 || it == P.maxiter) {  // true residual b - S x
      const double* y = product(x);
      if (!ok) break;
      double tr = 0.0, tz = 0.0;
      for (int j = t; j < n; j += C64_T) {
        const double rj = P.b[j] - y[j];
        r[j] = rj;
        const double r2 = rj * rj;
        tr += r2;
        tz = fma(w[j], r2, tz);
      }
      block_sums(tr, tz, true, n, s, [&](double, double v) { s.c = v / rz; });
      last = s.a;
      rzn = s.b;
      beta = s.c;
      if (converged(last)) {
        done = true;
        break;
      }
      if (guard) {
        const double rel = bnorm > 0 ? sqrt(last) / bnorm : 0.0;
        if (rel < best) {
          best = rel;
          stalled = 0;
          for (int i = t; i < nr; i += C64_T) P.x[r0 + i] = x[r0 + i];
        } else if (++stalled >= P.stall) {
          break;
        }
      }
    }
    rz = rzn;
    for (int j = t; j < n; j += C64_T) p[j] = fma(beta, p[j], r[j]);
    __syncthreads();
  }
  double relres = bnorm > 0 ? sqrt(last) / bnorm : 0.0;
  __syncthreads();
  if (guard && best < relres) relres = best;  // stopped past the best iterate: P.x holds it
  else
    for (int i = t; i < nr; i += C64_T) P.x[r0 + i] = x[r0 + i];
  if (rank == 0 && t == 0) {
    *P.iters = it;
    *P.relres = relres;
  }
  if (!GRID) cg::this_cluster().sync();  // shared memory stays until every CTA is done with it
}

// lanes per row: the fewest (of 4, 8, 16, 32) that keep at least 128 threads
// (a warp per scheduler) on the CTA's rows -- each doubling adds a shuffle
// stage of FP64 adds to every row
int lanes_per_row(int R) {
  int l = 4;
  while (l < 32 && R * l < 128) l *= 2;
  return l;
}

// stride of a resident row: l lanes of each row of a half-warp read l
// consecutive doubles, so rows l doubles apart (mod 16) use distinct banks
int slab_ld(int n, int l) {
  if (l >= 16) return n;
  int ld = n;
  while (ld % 16 != l) ++ld;
  return ld;
}

}  // namespace

namespace {

int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  return sms;
}

// rows per CTA, lanes per row and shared memory of one variant
size_t plan(const CG64Problem& P, bool grid, int G, CG64Args* A) {
  const bool csr = P.rowptr != nullptr;
  const int n = P.n;
  A->R = (n + G - 1) / G;
  A->lpr = lanes_per_row(A->R);
  A->ld = slab_ld(n, A->lpr);
  const size_t vecs = (size_t)(grid ? 5 : 6) * n * sizeof(double);
  const size_t slab = csr ? (size_t)cg64_csr_slab(P, A->R) * (sizeof(double) + sizeof(int))
                          : (size_t)A->R * A->ld * sizeof(double);
  A->resident = vecs + slab <= (size_t)C64_MAX_SMEM;
  A->slab_nnz = csr && A->resident ? cg64_csr_slab(P, A->R) : 0;
  return vecs + (A->resident ? slab : 0);
}

template <bool CSR>
int run_cluster(const CG64Args& A, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C64_CLUSTER);
  cfg.blockDim = dim3(C64_T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C64_CLUSTER;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  ILM_CHECK_CUDA(cudaLaunchKernelEx(&cfg, k_cg64<CSR, false>, A));
  return ILM_OK;
}

template <bool CSR>
int run_grid(CG64Args& A, int G, size_t smem, cudaStream_t st) {
  void* args[1] = {&A};
  ILM_CHECK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_cg64<CSR, true>), dim3(G), dim3(C64_T), args,
                                             smem, st));
  return ILM_OK;
}

template <bool CSR, bool GRID>
cudaError_t kernel_attributes() {
  const cudaError_t e = cudaFuncSetAttribute(k_cg64<CSR, GRID>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             C64_MAX_SMEM);
  if (e != cudaSuccess || GRID) return e;
  return cudaFuncSetAttribute(k_cg64<CSR, GRID>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

}  // namespace

// ---------------------------------------------------------------------------
// FP32 inverse of A = W S (symmetric; positive definite, or with one negative
// eigenvalue in the constant mode, as the Dirichlet Schur complement's net
// charge).  With E = 1^T W S 1 < 0, P = A + gamma w w^T, gamma = 2 |E| /
// (sum w)^2, is definite and A^-1 = P^-1 + kappa g g^T, g = P^-1 w, kappa =
// gamma / (1 - gamma w^T g).  Blocked Gauss-Jordan without pivoting on 32 x 32
// tiles, one launch per block column (each step reads one copy of the matrix
// and writes the other), w carried along as a right-hand side.  A pivot that
// is not positive marks the inverse unusable.  n = 157 / 448 / 696: 5 / 14 / 22
// launches.
// ---------------------------------------------------------------------------
namespace {

constexpr int GJ = 32;

// sums[j] = sum_i w_i S_ij (dense, a warp per column) or sum_e w_j S_je (CSR, a
// warp per row): both total 1^T W S 1
__global__ void __launch_bounds__(256) k_inv_sums(int n, const double* __restrict__ S, const int* __restrict__ rowptr,
                                                  const float* __restrict__ vhi, const float* __restrict__ vlo,
                                                  const double* __restrict__ w, double* __restrict__ sums) {
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (j >= n) return;
  double a = 0.0;
  if (rowptr) {
    for (int e = rowptr[j] + lane; e < rowptr[j + 1]; e += 32) a += (double)vhi[e] + (double)vlo[e];
    a *= w ? w[j] : 1.0;
  } else {
    for (int i = lane; i < n; i += 32) a = fma(w ? w[i] : 1.0, S[(size_t)j * n + i], a);
  }
  a = warp_sum(a);
  if (lane == 0) sums[j] = a;
}

// scalars: [0] usable, [1] kappa, [2] gamma, [3] not used
__global__ void __launch_bounds__(1024) k_inv_shift(int n, const double* __restrict__ sums,
                                                    const double* __restrict__ w, float* __restrict__ sc) {
  __shared__ double ra[32], rb[32];
  double a = 0.0, b = 0.0;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    a += sums[j];
    b += w ? w[j] : 1.0;
  }
  a = warp_sum(a);
  b = warp_sum(b);
  if ((threadIdx.x & 31) == 0) {
    ra[threadIdx.x >> 5] = a;
    rb[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = b = 0.0;
    for (int k = 0; k < 32; ++k) {
      a += ra[k];
      b += rb[k];
    }
    sc[0] = 1.f;
    sc[1] = 0.f;
    sc[2] = a < 0.0 ? (float)(-2.0 * a / (b * b)) : 0.f;
  }
}

// tiles of P (identity in the padding), transposed (P is symmetric), and w
__global__ void __launch_bounds__(256) k_inv_form(int n, int ld, const double* __restrict__ S,
                                                  const double* __restrict__ w, const float* __restrict__ sc,
                                                  float* __restrict__ T) {
  const int j = blockIdx.x * 32 + (threadIdx.x & 31), i = blockIdx.y * 8 + (threadIdx.x >> 5), np = ld - GJ;
  if (i >= np || j >= ld) return;
  double v = 0.0;
  const double gamma = (double)sc[2];
  if (j >= np) {
    v = j == np && i < n ? (w ? w[i] : 1.0) : 0.0;
  } else if (i < n && j < n) {
    const double wj = w ? w[j] : 1.0, wi = w ? w[i] : 1.0;
    v = gamma * wi * wj;
    if (S) v = fma(wj, S[(size_t)i * n + j], v);
  } else {
    v = i == j ? 1.0 : 0.0;
  }
  T[(size_t)i * ld + j] = (float)v;
}

__global__ void k_inv_form_csr(int n, int ld, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                               const float* __restrict__ vhi, const float* __restrict__ vlo,
                               const double* __restrict__ w, float* __restrict__ T) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) return;
  const double wi = w ? w[i] : 1.0;
  for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32)
    T[(size_t)i * ld + colidx[e]] += (float)(wi * ((double)vhi[e] + (double)vlo[e]));
}

// M <- M^-1 in place, 256 threads (thread: row t / 8, four columns)
__device__ __forceinline__ void invert_tile(float (*M)[GJ + 1], float* __restrict__ sc) {
  const int r = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 4;
  for (int s = 0; s < GJ; ++s) {
    __syncthreads();
    float p = M[s][s];
    if (!(p > 0.f) || !(p < 3e38f)) {
      if (threadIdx.x == 0) sc[0] = 0.f;
      p = 1.f;
    }
    const float ip = 1.f / p, f = M[r][s] * ip;
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = c0 + q;
      const float u = c == s ? 1.f : M[s][c];
      v[q] = r == s ? u * ip : fmaf(-f, u, c == s ? 0.f : M[r][c]);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) M[r][c0 + q] = v[q];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) k_inv_diag(int ld, const float* __restrict__ T, float* __restrict__ D,
                                                  float* __restrict__ sc) {
  __shared__ float M[GJ][GJ + 1];
  const int r = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 4;
  for (int q = 0; q < 4; ++q) M[r][c0 + q] = T[(size_t)r * ld + c0 + q];
  invert_tile(M, sc);
  for (int q = 0; q < 4; ++q) D[r * GJ + c0 + q] = M[r][c0 + q];
}

// one block column: B = the matrix after eliminating block k of A (D: the
// inverse of A's diagonal block k); the CTA of block k + 1 inverts its result
__global__ void __launch_bounds__(256) k_inv_step(int k, int ld, const float* __restrict__ A, float* __restrict__ B,
                                                  const float* __restrict__ D, float* __restrict__ Dn,
                                                  float* __restrict__ sc) {
  __shared__ float d[GJ][GJ + 1], l[GJ][GJ + 1], u[GJ][GJ + 1], m[GJ][GJ + 1];
  const int bi = blockIdx.y, bj = blockIdx.x, r = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 4;
  pdl_wait();
  const size_t at = (size_t)(bi * GJ + r) * ld + bj * GJ + c0;
  float v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    d[r][c0 + q] = D[r * GJ + c0 + q];
    l[r][c0 + q] = A[(size_t)(bi * GJ + r) * ld + k * GJ + c0 + q];
    u[r][c0 + q] = A[(size_t)(k * GJ + r) * ld + bj * GJ + c0 + q];
    v[q] = bi == k || bj == k ? 0.f : A[at + q];
  }
  __syncthreads();
  if (bj == k) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float a = 0.f;
      for (int e = 0; e < GJ; ++e) a = fmaf(l[r][e], d[e][c0 + q], a);
      v[q] = bi == k ? d[r][c0 + q] : -a;
    }
  } else {
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    for (int e = 0; e < GJ; ++e)
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = fmaf(d[r][e], u[e][c0 + q], x[q]);
    if (bi == k) {
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = x[q];
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) m[r][c0 + q] = x[q];
      __syncthreads();
      for (int e = 0; e < GJ; ++e)
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = fmaf(-l[r][e], m[e][c0 + q], v[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) B[at + q] = v[q];
  if (bi == k + 1 && bj == k + 1 && (k + 2) * GJ <= ld) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) m[r][c0 + q] = v[q];
    invert_tile(m, sc);
#pragma unroll
    for (int q = 0; q < 4; ++q) Dn[r * GJ + c0 + q] = m[r][c0 + q];
  }
}

// kappa of the shift
__global__ void __launch_bounds__(1024) k_inv_kappa(int n, int ld, const float* __restrict__ T,
                                                    const double* __restrict__ w, float* __restrict__ sc) {
  __shared__ double ra[32];
  double a = 0.0;
  for (int j = threadIdx.x; j < n; j += blockDim.x) a += (w ? w[j] : 1.0) * (double)T[(size_t)j * ld + ld - GJ];
  a = warp_sum(a);
  if ((threadIdx.x & 31) == 0) ra[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    a = 0.0;
    for (int k = 0; k < 32; ++k) a += ra[k];
    const double gamma = (double)sc[2], q = 1.0 - gamma * a;
    if (gamma != 0.0) {
      sc[1] = (float)(gamma / q);
      if (!(fabs(q) > 1e-3)) sc[0] = 0.f;
    }
  }
}

}  // namespace

int cg64_inverse(CG64Inverse* I, const CG64Problem& P, cudaStream_t st) {
  const int n = P.n, nt = (n + GJ - 1) / GJ, ld = nt * GJ + GJ;
  const size_t bytes = (size_t)nt * GJ * ld * sizeof(float);
  ILM_TRY(I->a.alloc(bytes));
  ILM_TRY(I->b.alloc(bytes));
  // scalars, two diagonal blocks, FP64 sums
  ILM_TRY(I->s.alloc((4 + 2 * GJ * GJ) * sizeof(float) + (size_t)n * sizeof(double)));
  float* sc = I->s.as<float>();
  float* D[2] = {sc + 4, sc + 4 + GJ * GJ};
  double* sums = reinterpret_cast<double*>(sc + 4 + 2 * GJ * GJ);
  float* T[2] = {I->a.as<float>(), I->b.as<float>()};
  k_inv_sums<<<(n * 32 + 255) / 256, 256, 0, st>>>(n, P.A, P.rowptr, P.vhi, P.vlo, P.w, sums);
  ILM_CHECK_LAUNCH();
  k_inv_shift<<<1, 1024, 0, st>>>(n, sums, P.w, sc);
  ILM_CHECK_LAUNCH();
  k_inv_form<<<dim3(ld / 32, nt * GJ / 8), 256, 0, st>>>(n, ld, P.rowptr ? nullptr : P.A, P.w, sc, T[0]);
  ILM_CHECK_LAUNCH();
  if (P.rowptr) {
    k_inv_form_csr<<<(n * 32 + 255) / 256, 256, 0, st>>>(n, ld, P.rowptr, P.colidx, P.vhi, P.vlo, P.w, T[0]);
    ILM_CHECK_LAUNCH();
  }
  k_inv_diag<<<1, 256, 0, st>>>(ld, T[0], D[0], sc);
  ILM_CHECK_LAUNCH();
  for (int k = 0; k < nt; ++k)
    ILM_CHECK_CUDA(launch_pdl(k_inv_step, dim3(nt + 1, nt), dim3(256), st, k, ld, (const float*)T[k & 1], T[(k + 1) & 1],
                              (const float*)D[k & 1], D[(k + 1) & 1], sc));
  k_inv_kappa<<<1, 1024, 0, st>>>(n, ld, T[nt & 1], P.w, sc);
  ILM_CHECK_LAUNCH();
  I->n = n;
  I->ld = ld;
  I->inv = T[nt & 1];
  I->ready = true;
  return ILM_OK;
}

size_t cg64_scratch_bytes(int n) { return sizeof(CG64State) + 2 * (size_t)n * sizeof(double); }

bool cg64_fits(int n) { return 5 * (size_t)n * sizeof(double) + 384 <= (size_t)227 * 1024; }

int launch_cg64(const CG64Problem& P, void* scratch, cudaStream_t st, int variant) {
  const int n = P.n;
  if (!cg64_fits(n)) {
    set_error("CG: problem of %d unknowns exceeds the shared-memory solver", n);
    return ILM_ERR_SIZE_LIMIT;
  }
  const bool csr = P.rowptr != nullptr;
  CG64Args A;
  A.p = P;
  A.state = static_cast<CG64State*>(scratch);
  A.gq = reinterpret_cast<double*>(A.state + 1);
  if (!A.p.iters) A.p.iters = &A.state->iters;
  if (!A.p.relres) A.p.relres = &A.state->relres;
  ILM_CHECK_CUDA(cudaMemsetAsync(A.state, 0, sizeof(CG64State), st));
  if (!A.p.timeout) A.p.timeout = &A.state->timeout;
  const long long entries = (long long)n * (csr ? std::min(P.max_row_nnz, n) : n);
  size_t smem = plan(P, false, C64_CLUSTER, &A);
  if ((variant == 1 || (variant == 0 && entries <= C64_CLUSTER_ENTRIES)) && smem <= (size_t)C64_MAX_SMEM &&
      (csr || A.resident)) {
    ILM_CHECK_CUDA((csr ? kernel_attributes<true, false>() : kernel_attributes<false, false>()));
    return csr ? run_cluster<true>(A, smem, st) : run_cluster<false>(A, smem, st);
  }
  const int sms = device_sms();
  if (sms < 1) {
    set_error("CG: no device");
    return ILM_ERR_CUDA;
  }
  smem = plan(P, true, std::min(sms, n), &A);
  ILM_CHECK_CUDA((csr ? kernel_attributes<true, true>() : kernel_attributes<false, true>()));
  const int G = (n + A.R - 1) / A.R;
  return csr ? run_grid<true>(A, G, smem, st) : run_grid<false>(A, G, smem, st);
}

}  // namespace ilm
