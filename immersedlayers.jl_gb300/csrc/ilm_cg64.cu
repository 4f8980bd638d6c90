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
// step gains less than a factor of four the CG goes on from there.  The
// correction that follows the residual that passes stays if its own residual
// passes too (that is the one reported), else it is taken back.
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
#include <utility>

#include "ilm_internal.cuh"

namespace cg = cooperative_groups;

namespace ilm {
namespace {

constexpr int C64_T = 256;             // threads per CTA
constexpr int C64_CLUSTER = 16;        // CTAs of the cluster variant
// dynamic shared memory beside the static scalars
constexpr int C64_MAX_CLUSTER = 227 * 1024 - 512, C64_MAX_GRID = 227 * 1024 - 256;
// matrix entries up to which the cluster variant is used without an FP32
// inverse (no memory for it): an iteration of a
// dense n takes 4.8 / 5.4 / 6.9 / 8.2 us with the cluster and 5.5 / 5.8 / 6.8 /
// 6.9 us with the grid at n = 157 / 224 / 300 / 400
constexpr long long C64_CLUSTER_ENTRIES = 256 * 256;
// unknowns up to which it is used with an FP32 inverse, whose rows 16 SMs read
// from L2 (us per solve, cluster and grid: dense n = 157 25 / 33, 300 39.6 /
// 41.2, 400 41.6 / 34.9; 19 entries a row, n = 157 29 / 39, 560 39.1 / 39.8,
// 696 43.3 / 41.3; both about 1 us more since the last correction is judged)
constexpr int C64_CLUSTER_DENSE = 320, C64_CLUSTER_CSR = 560;
constexpr unsigned C64_SPIN = 1u << 22;  // polls of the grid barrier before it gives up (seconds)

struct CG64Args {
  CG64Problem p;
  int R;            // rows per CTA
  int lpr;          // lanes per row of the product (4, 8, 16, 32)
  int resident;     // the CTA's rows of S are kept in shared memory
  int ld;           // row stride of the resident dense slab (doubles)
  int slab_nnz;     // CSR: entries of the largest slab
  int nv;           // stride of the shared-memory vectors (n rounded up to 4)
  double* gq;       // grid variant: exchange (two vectors of n doubles, three sums per CTA)
  CG64State* state;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// shared-memory scalars: [0, 8) and [8, 16) warp partials, then the results
struct Scal {
  double part[C64_CLUSTER];
  float part32[8];
  double a, b, c;   // first sum, second sum, derived scalar
  unsigned top;     // refinement: largest magnitude bits of b
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
  double* r = x + A.nv;
  double* p = r + A.nv;
  double* w = p + A.nv;
  double* qb = w + A.nv;                       // cluster: two buffers; grid: one
  double* slab = qb + (GRID ? 1 : 2) * (size_t)A.nv;
  int* scol = reinterpret_cast<int*>(slab + A.slab_nnz);
  __shared__ Scal s;
  __shared__ int s_ok;
  __shared__ double tot[GRID ? 1 : 2 * C64_CLUSTER];  // refinement: the CTAs' parts of |r|^2 and |b|^2
  int par = 0;           // exchange buffer
  unsigned bar = 0;      // grid barriers passed
  bool ok = true;

  int e0 = 0;
  if (CSR) e0 = P.rowptr[r0];
  if (A.resident) {
    if (CSR) {
      const int e1 = P.rowptr[r0 + nr];
      for (int e = e0 + t; e < e1; e += C64_T) {
        slab[e - e0] = widen(P.vhi[e]) + widen(P.vlo[e]);
        scol[e - e0] = P.colidx[e];
      }
    } else {
      for (int k = t; k < nr * n; k += C64_T) {
        const int j = k / nr, i = k - j * nr;
        slab[(size_t)i * A.ld + j] = P.A[(size_t)j * n + r0 + i];
      }
    }
  }

  // what the CTAs sent becomes visible to all
  auto barrier = [&]() {
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
    } else {
      cg::this_cluster().sync();
    }
  };

  // the CTAs' rows of one vector become visible to all
  auto publish = [&](double* q) {
    barrier();
    if (GRID)
      for (int j = t; j < n; j += C64_T) q[j] = __ldcg(A.gq + (size_t)par * n + j);
    // no CTA barrier here: each thread reads back the entries it stored
    par ^= 1;
  };

  // rows r0 .. r0 + nr of S v; emit(i, value, c, L) with row i's value in each
  // of its L lanes (c: the lane)
  auto rows_of = [&](const double* v, auto emit) {
    const int L = A.lpr, c = t & (L - 1), rows = C64_T / L;
    if (!CSR && GRID && !A.resident) {
      // S streamed from L2: consecutive threads take consecutive rows of one
      // column, partial sums meet in qb (free between products; n > C64_T here)
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
          qb[t] = a0 + a1;
        }
        __syncthreads();
        if (t < m) {
          double a = qb[t];
          for (int u = 1; u < nc; ++u) a += qb[u * m + t];
          emit(b0 + t, a, 0, 1);
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
                a0 = fma(widen(__ldg(P.vhi + k)) + widen(__ldg(P.vlo + k)), v[__ldg(P.colidx + k)], a0);
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
        if (i < nr) emit(i, a0, c, L);
      }
    }
  };

  // entry k (of this CTA's rows, or any) of an exchanged vector, to every CTA
  auto send = [&](double* local, double* global, int k, double v, int c, int L) {
    if (GRID) {
      if (c == 0) __stcg(global + k, v);
    } else {
      for (int d = c; d < G; d += L) cg::this_cluster().map_shared_rank(local, d)[k] = v;
    }
  };

  // S v in all CTAs (cluster: the buffer the other CTAs wrote; grid: the CTA's own copy)
  auto product = [&](const double* v) -> double* {
    double* q = GRID ? qb : qb + (size_t)par * A.nv;
    rows_of(v, [&](int i, double a, int c, int L) { send(q, A.gq + (size_t)par * n, r0 + i, a, c, L); });
    publish(q);
    return q;
  };

  for (int j = t; j < n; j += C64_T) {
    x[j] = P.x0 ? P.x0[j] : 0.0;
    w[j] = P.w ? P.w[j] : 1.0;
  }
  if (!GRID) cg::this_cluster().sync();  // every CTA of the cluster runs before its shared memory is written
  __syncthreads();
  double bb = 0.0, rr = 0.0, bnorm = 0.0, thr2 = 0.0, thr = 0.0, last = 0.0;
  auto set_norm = [&]() {
    bnorm = sqrt(bb);
    thr = P.tol * bnorm;
    thr2 = thr * thr;
    last = bb;
  };
  // squared norms are compared, except where they are about to underflow
  auto below = [&](double v) { return v <= thr2 || v < 1e-280; };
  auto converged = [&](double v) { return thr2 > 1e-280 ? v <= thr2 : sqrt(v) <= thr; };
  // r = b - S x0, or b (x0 may be the output: all CTAs have read it at the barrier)
  auto start = [&]() {
    const double* q = P.x0 ? product(x) : nullptr;
    for (int j = t; j < n; j += C64_T) r[j] = P.x0 ? P.b[j] - q[j] : P.b[j];
  };
  int it = 0;
  bool done = false;
  const bool refine = P.inv && P.invs[0] != 0.f;
  if (refine) {
    // Steps x += P r, r = b - S x.  A CTA forms r and the update of x for its own
    // rows only (a pass of FP64 operations over all n costs n / 1.7 clocks) and
    // sends W r, in FP32, and x: two barriers per step.  The norm of a residual is
    // summed beside the product with P and judged beside the next residual's, by
    // the last warp, off the chain of the others: so the correction after the
    // residual that passes is always taken, and its residual is there.  It is
    // wanted: the residual that passes is rich in the modes that P gets least right,
    // the slow ones, and x is further off for it than a CG iterate of that residual.
    // Nothing says that P contracts on it, so its residual decides (about 1 us of
    // a solve).
    float* v = reinterpret_cast<float*>(p);               // W r scaled into FP32's range
    float* gv = reinterpret_cast<float*>(A.gq + n);       // grid: its exchange
    double* gs = A.gq + 2 * (size_t)n;                    // grid: the CTAs' sums (three each)
    const int lane = t & 31, warp = t >> 5;
    const float kappa = P.invs[1];
    if (t == 0) s.top = 0u;
    __syncthreads();
    unsigned top = 0u;
    for (int j = t; j < n; j += C64_T) top = max(top, (unsigned)__double2hiint(P.b[j]) & 0x7fffffffu);
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) atomicMax(&s.top, top);
    for (int j = n + t; j < A.nv; j += C64_T) v[j] = 0.f;
    __syncthreads();
    const int e = min(max((int)(s.top >> 20) - 1023, -1000), 1000);  // max |b| ~ 2^e
    const double down = __hiloint2double((1023 - e) << 20, 0), up = __hiloint2double((1023 + e) << 20, 0);
    auto residual = [&](int i, double y, int c, int L) {
      const double ri = P.b[r0 + i] - y;
      const float vi = (float)(w[r0 + i] * (ri * down));
      if (c == 0) r[r0 + i] = ri;
      if (GRID) {
        if (c == 0) __stcg(gv + r0 + i, vi);
      } else {
        for (int d = c; d < G; d += L) cg::this_cluster().map_shared_rank(v, d)[r0 + i] = vi;
      }
    };
    auto gather_x = [&]() {
      if (GRID)
        for (int j = t; j < n; j += C64_T) x[j] = __ldcg(A.gq + j);
      __syncthreads();
    };
    constexpr int LAST = C64_T / 32 - 1;
    enum { DONE = 1, UNDO = 2, RESET = 4 };
    double* old = p + A.nv / 2;  // the CTA's rows of x before the last correction (behind v)
    int flags = 0;
    if (!P.x0)
      for (int i = t; i < nr; i += C64_T) residual(i, 0.0, 0, 1);
    for (int round = 0;; ++round) {
      if (round || P.x0) rows_of(x, residual);
      if (round && warp == LAST) {  // judge the residual of the round before
        double a = 0.0, b = 0.0;
        for (int k = lane; k < G; k += 32) {
          a += GRID ? __ldcg(gs + 2 * k) : tot[2 * k];
          if (round == 1) b += GRID ? __ldcg(gs + 2 * k + 1) : tot[2 * k + 1];
        }
        const double now = warp_sum(a);
        int f = 0;
        if (round == 1) {
          bb = warp_sum(b);
          rr = now;
          set_norm();
          last = rr;
          if (bnorm == 0.0 || rr == 0.0) f = DONE | UNDO;
          else if (converged(rr)) f = DONE;
        } else {
          if (converged(now)) f |= DONE;
          if (!(now <= 0.0625 * last)) f |= UNDO;                   // slow: from here on CG
          if (f == UNDO && !(now <= rr)) f |= RESET;                // no better than the start: the CG begins there
          last = f & RESET ? rr : now;
        }
        if (f == 0 && round - 1 >= P.maxiter) f = UNDO;
        if (lane == 0) {
          s.a = last;
          s.b = bb;
          s.flag = f;
        }
      }
      __syncthreads();
      if (round) {
        it = round - 1;
        flags = s.flag;
        if (flags) break;
      }
      barrier();
      if (!ok) break;
      if (GRID)
        for (int j = t; j < n; j += C64_T) v[j] = __ldcg(gv + j);
      float shift = 0.f;
      if (kappa != 0.f) {
        float g = 0.f;
        for (int j = t; j < n; j += C64_T) g = fmaf(__ldg(P.invg + j), v[j], g);
        for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
        if (lane == 0) s.part32[warp] = g;
      }
      __syncthreads();
      if (kappa != 0.f) {
        for (int k = 0; k < C64_T / 32; ++k) shift += s.part32[k];
        shift *= kappa;
      }
      // rows of P v, each a warp's (the last warp takes its CTA's part of the norms first)
      if (warp == LAST) {
        double a = 0.0, b = 0.0;
        for (int i = lane; i < nr; i += 32) {
          a = fma(r[r0 + i], r[r0 + i], a);
          if (round == 0) b = fma(P.b[r0 + i], P.b[r0 + i], b);
        }
        a = warp_sum(a);
        send(tot, gs, 2 * rank, a, lane, 32);
        if (round == 0) {
          b = warp_sum(b);
          send(tot, gs, 2 * rank + 1, b, lane, 32);
        }
      }
      const float4* v4 = reinterpret_cast<const float4*>(v);
      const int n4 = A.nv / 4;
      for (int i = warp; i < nr; i += C64_T / 32) {
        const float4* row = reinterpret_cast<const float4*>(P.inv + (size_t)(r0 + i) * P.ldi);
        float a[4] = {0.f, 0.f, 0.f, 0.f};
        for (int j0 = 0; j0 < n4; j0 += 4 * 32) {  // four 16-byte loads from L2 in flight
          float4 m[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int j = j0 + 32 * q + lane;
            m[q] = j < n4 ? __ldg(row + j) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int j = j0 + 32 * q + lane;
            const float4 f = j < n4 ? v4[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            a[0] = fmaf(m[q].x, f.x, a[0]);
            a[1] = fmaf(m[q].y, f.y, a[1]);
            a[2] = fmaf(m[q].z, f.z, a[2]);
            a[3] = fmaf(m[q].w, f.w, a[3]);
          }
        }
        float u = (a[0] + a[1]) + (a[2] + a[3]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) u += __shfl_xor_sync(0xffffffffu, u, o);
        u = kappa != 0.f ? fmaf(shift, __ldg(P.invg + r0 + i), u) : u;
        const double x0 = x[r0 + i], xi = fma((double)u, up, x0);
        __syncwarp();  // every lane has read x before it is replaced
        if (lane == 0) old[i] = x0;
        send(x, A.gq, r0 + i, xi, lane, 32);
      }
      barrier();
      if (!ok) break;
      gather_x();
    }
    if (ok && flags == DONE) {
      // the residual of the x that has had one correction more (other CTAs may
      // still read the sums of the round before: not through tot)
      if (warp == LAST) {
        double a = 0.0;
        for (int i = lane; i < nr; i += 32) a = fma(r[r0 + i], r[r0 + i], a);
        send(s.part, gs + 2 * G, rank, warp_sum(a), lane, 32);
      }
      for (int i = t; i < nr; i += C64_T) {
        P.x[r0 + i] = x[r0 + i];
        if (GRID) __stcg(A.gq + n + r0 + i, old[i]);
      }
      if (GRID) {  // no CTA waits: the last to arrive decides for all rows
        __syncthreads();
        if (t == 0) {
          __threadfence();
          s_ok = atomicAdd(&A.state->finished, 1u) + 1 == (unsigned)G;
          __threadfence();
        }
        __syncthreads();
        if (!s_ok) return;
      } else {     // every CTA decides for its own
        barrier();
      }
      if (warp == LAST) {
        double a = 0.0;
        for (int k = lane; k < G; k += 32) a += GRID ? __ldcg(gs + 2 * G + k) : s.part[k];
        a = warp_sum(a);
        const bool keep = converged(a);
        if (!keep) {
          if (GRID)
            for (int j = lane; j < n; j += 32) P.x[j] = __ldcg(A.gq + n + j);
          else
            for (int i = lane; i < nr; i += 32) P.x[r0 + i] = old[i];
        }
        if ((GRID || rank == 0) && lane == 0) {
          *P.iters = it;
          *P.relres = fmin(sqrt((keep ? a : last) / bb), P.tol);
        }
      }
      return;  // (nothing more is written to another CTA)
    }
    if (ok) {
      done = flags & DONE;
      last = s.a;
      bb = s.b;
    }
    if (ok && flags & UNDO) {  // the last correction does not count
      barrier();
      for (int i = t; i < nr; i += C64_T)
        send(x, A.gq, r0 + i, flags & RESET ? (P.x0 ? P.x0[r0 + i] : 0.0) : old[i], 0, 1);
      barrier();
      gather_x();
    }
    if (ok && !done) {
      const double l = last;
      set_norm();
      last = l;
      par = 1;  // (others may still read the first exchange buffer)
      const double* y = product(x);
      for (int j = t; j < n; j += C64_T) r[j] = P.b[j] - y[j];
    }
    if (!ok) done = true;
  } else {
    start();
    for (int j = t; j < n; j += C64_T) {
      bb += P.b[j] * P.b[j];
      rr += r[j] * r[j];
    }
    block_sums(bb, rr, true, n, s, [](double, double) {});
    bb = s.a;
    rr = s.b;
    set_norm();
    done = bnorm == 0.0;
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
    if (!(fabs(s.a) > 0.0)) break;  // zero, or not a number
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
      s.flag = below(u) || !(u <= 1.7e308);
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
      if (!(last <= 1.7e308)) break;  // not a number
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
  double relres = 0.0;
  if (guard || (rank == 0 && t == 0)) relres = bb == 0.0 ? 0.0 : sqrt(last / bb);  // (data that are no numbers: NaN)
  if (done) relres = fmin(relres, P.tol);  // (squares were compared)
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
  A->nv = (n + 3) / 4 * 4;
  const size_t vecs = (size_t)(grid ? 5 : 6) * A->nv * sizeof(double);
  const size_t slab = csr ? (size_t)cg64_csr_slab(P, A->R) * (sizeof(double) + sizeof(int))
                          : (size_t)A->R * A->ld * sizeof(double);
  A->resident = vecs + slab <= (size_t)(grid ? C64_MAX_GRID : C64_MAX_CLUSTER);
  A->slab_nnz = csr && A->resident ? cg64_csr_slab(P, A->R) : 0;
  return vecs + (A->resident ? slab : 0);
}

template <bool CSR>
cudaError_t run_cluster(const CG64Args& A, size_t smem, cudaStream_t st) {
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
  return cudaLaunchKernelEx(&cfg, k_cg64<CSR, false>, A);
}

template <bool CSR>
cudaError_t run_grid(CG64Args& A, int G, size_t smem, cudaStream_t st) {
  void* args[1] = {&A};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_cg64<CSR, true>), dim3(G), dim3(C64_T), args, smem, st);
}

// a launch that the device (a partition of it, or a context limited to some of
// its SMs) has no room for
bool no_room(cudaError_t e) {
  return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorInvalidClusterSize ||
         e == cudaErrorLaunchOutOfResources || e == cudaErrorInvalidConfiguration || e == cudaErrorNotSupported;
}

template <bool CSR, bool GRID>
cudaError_t kernel_attributes() {
  const cudaError_t e = cudaFuncSetAttribute(k_cg64<CSR, GRID>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             GRID ? C64_MAX_GRID : C64_MAX_CLUSTER);
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
// launches, 47 / 112 / 191 us.
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

constexpr int GJL = GJ + 4;  // row stride of a tile in shared memory (16-byte rows)

// M <- M^-1 in place (M symmetric) by the first warp.  A lane holds a column in
// registers, rotated so that the pivot's row is always the first (a rolled loop:
// 32 unrolled steps run once each are bound by instruction fetch, 6 us); the
// pivot column is the pivot row, negative where the pivots are done, and goes
// through shared memory; the next pivot's row comes first, its reciprocal (with
// one Newton step) runs beside the other rows.  3.7 us, a chain of latencies; 256
// threads on the tile in shared memory, two CTA barriers and an IEEE division
// per pivot, took 8 us.
__device__ __forceinline__ void invert_tile(float (*M)[GJL], float (*col)[GJ], float* __restrict__ sc) {
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    bool bad = false;
    float a[GJ];
#pragma unroll
    for (int r = 0; r < GJ; ++r) a[r] = M[r][lane];
    float p = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll 1
    for (int s = 0; s < GJ; ++s) {
      float* c = col[s & 1];
      c[(lane - s) & 31] = lane < s ? -a[0] : a[0];
      const bool mine = lane == s;
      bad |= !(p > 0.f) || !(p < 3e38f);
      float ip = __fdividef(1.f, p);
      ip = fmaf(ip, fmaf(-p, ip, 1.f), ip);
      const float u = mine ? ip : a[0] * ip;
      __syncwarp();
#pragma unroll
      for (int r = 0; r < GJ; r += 4) {
        const float4 f = *reinterpret_cast<const float4*>(c + r);
        if (r) a[r - 1] = fmaf(-f.x, u, mine ? 0.f : a[r]);
        a[r] = fmaf(-f.y, u, mine ? 0.f : a[r + 1]);
        if (r == 0) p = __shfl_sync(0xffffffffu, a[0], (s + 1) & 31);
        a[r + 1] = fmaf(-f.z, u, mine ? 0.f : a[r + 2]);
        a[r + 2] = fmaf(-f.w, u, mine ? 0.f : a[r + 3]);
      }
      a[GJ - 1] = u;
    }
    if (bad) sc[0] = 0.f;
#pragma unroll
    for (int r = 0; r < GJ; ++r) M[r][lane] = a[r];
  }
  __syncthreads();
}

// acc += sign * (row r of X) Y, four columns from c0
__device__ __forceinline__ void tile_mm(float4& acc, float sign, const float (*X)[GJL], const float (*Y)[GJL], int r,
                                        int c0) {
#pragma unroll
  for (int e = 0; e < GJ; e += 4) {
    const float4 x4 = *reinterpret_cast<const float4*>(&X[r][e]);
    const float x[4] = {sign * x4.x, sign * x4.y, sign * x4.z, sign * x4.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 y = *reinterpret_cast<const float4*>(&Y[e + q][c0]);
      acc.x = fmaf(x[q], y.x, acc.x);
      acc.y = fmaf(x[q], y.y, acc.y);
      acc.z = fmaf(x[q], y.z, acc.z);
      acc.w = fmaf(x[q], y.w, acc.w);
    }
  }
}

__device__ __forceinline__ float4& at4(float* p) { return *reinterpret_cast<float4*>(p); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

__global__ void __launch_bounds__(256) k_inv_diag(int ld, const float* __restrict__ T, float* __restrict__ D,
                                                  float* __restrict__ sc) {
  __shared__ __align__(16) float M[GJ][GJL], col[2][GJ];
  const int r = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 4;
  at4(&M[r][c0]) = ld4(T + (size_t)r * ld + c0);
  invert_tile(M, col, sc);
  at4(D + r * GJ + c0) = at4(&M[r][c0]);
}

// one block column: B = the matrix after eliminating block k of A (D: the
// inverse of A's diagonal block k); the CTA of block k + 1 (the first, so that
// the others run beside it) inverts its result
__global__ void __launch_bounds__(256) k_inv_step(int k, int nt, int ld, const float* __restrict__ A,
                                                  float* __restrict__ B, const float* __restrict__ D,
                                                  float* __restrict__ Dn, float* __restrict__ sc) {
  __shared__ __align__(16) float d[GJ][GJL], l[GJ][GJL], u[GJ][GJL], m[GJ][GJL], col[2][GJ];
  const int next = k + 1 < nt ? (k + 1) * (nt + 1) + k + 1 : 0;
  const int tile = blockIdx.x == 0 ? next : blockIdx.x == next ? 0 : blockIdx.x;
  const int bi = tile / (nt + 1), bj = tile - bi * (nt + 1), r = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 4;
  pdl_wait();
  const size_t at = (size_t)(bi * GJ + r) * ld + bj * GJ + c0;
  const bool fresh = bi == k || bj == k;
  const float4 dv = ld4(D + r * GJ + c0), lv = ld4(A + (size_t)(bi * GJ + r) * ld + k * GJ + c0),
               uv = ld4(A + (size_t)(k * GJ + r) * ld + bj * GJ + c0);
  float4 v = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4(A + at);
  at4(&d[r][c0]) = dv;
  at4(&l[r][c0]) = lv;
  at4(&u[r][c0]) = uv;
  __syncthreads();
  if (bj == k) {
    if (bi == k) v = dv;
    else tile_mm(v, -1.f, l, d, r, c0);
  } else if (bi == k) {
    tile_mm(v, 1.f, d, u, r, c0);
  } else {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    tile_mm(x, 1.f, d, u, r, c0);
    at4(&m[r][c0]) = x;
    __syncthreads();
    tile_mm(v, -1.f, l, m, r, c0);
  }
  at4(B + at) = v;
  if (bi == k + 1 && bj == k + 1) {
    at4(&u[r][c0]) = v;
    invert_tile(u, col, sc);
    at4(Dn + r * GJ + c0) = at4(&u[r][c0]);
  }
}

// kappa of the shift; g = P^-1 w as one vector
__global__ void __launch_bounds__(1024) k_inv_kappa(int n, int ld, const float* __restrict__ T,
                                                    const double* __restrict__ w, float* __restrict__ sc,
                                                    float* __restrict__ g) {
  __shared__ double ra[32];
  double a = 0.0;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    g[j] = T[(size_t)j * ld + ld - GJ];
    a += (w ? w[j] : 1.0) * (double)g[j];
  }
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

int cg64_inverse(CG64Inverse* I, DevBuf* tmp, const CG64Problem& P, cudaStream_t st) {
  const int n = P.n, nt = (n + GJ - 1) / GJ, ld = nt * GJ + GJ;
  const size_t bytes = (size_t)nt * GJ * ld * sizeof(float);
  I->ready = false;
  // (scalars, two diagonal blocks, FP64 sums in s)
  if (I->a.alloc(bytes) != ILM_OK || tmp->alloc(bytes) != ILM_OK ||
      I->s.alloc((4 + 2 * GJ * GJ) * sizeof(float) + (size_t)n * sizeof(double)) != ILM_OK) {
    (void)cudaGetLastError();
    I->a.release();
    return ILM_OK;
  }
  float* sc = I->s.as<float>();
  float* D[2] = {sc + 4, sc + 4 + GJ * GJ};
  double* sums = reinterpret_cast<double*>(sc + 4 + 2 * GJ * GJ);
  float* T[2] = {I->a.as<float>(), tmp->as<float>()};
  if (nt & 1) std::swap(T[0], T[1]);  // the last step writes a
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
    ILM_CHECK_CUDA(launch_pdl(k_inv_step, dim3((nt + 1) * nt), dim3(256), st, k, nt, ld, (const float*)T[k & 1], T[(k + 1) & 1],
                              (const float*)D[k & 1], D[(k + 1) & 1], sc));
  k_inv_kappa<<<1, 1024, 0, st>>>(n, ld, T[nt & 1], P.w, sc, reinterpret_cast<float*>(sums));
  ILM_CHECK_LAUNCH();
  I->n = n;
  I->ld = ld;
  I->g = reinterpret_cast<float*>(sums);
  I->ready = true;
  return ILM_OK;
}

size_t cg64_scratch_bytes(int n) { return sizeof(CG64State) + 5 * (size_t)n * sizeof(double); }

bool cg64_fits(int n) { return 5 * (size_t)((n + 3) / 4 * 4) * sizeof(double) <= (size_t)C64_MAX_GRID; }

int launch_cg64(const CG64Problem& P, void* scratch, cudaStream_t st) {
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
  const bool few = P.inv ? n <= (csr ? C64_CLUSTER_CSR : C64_CLUSTER_DENSE) : entries <= C64_CLUSTER_ENTRIES;
  if (few && smem <= (size_t)C64_MAX_CLUSTER && (csr || A.resident)) {
    cudaError_t e = csr ? kernel_attributes<true, false>() : kernel_attributes<false, false>();
    if (e == cudaSuccess) e = csr ? run_cluster<true>(A, smem, st) : run_cluster<false>(A, smem, st);
    if (!no_room(e)) {
      ILM_CHECK_CUDA(e);
      return ILM_OK;
    }
    (void)cudaGetLastError();
  }
  ILM_CHECK_CUDA((csr ? kernel_attributes<true, true>() : kernel_attributes<false, true>()));
  // a CTA per SM; where they cannot all be resident, half as many, down to four (at
  // which 256 unknowns still fit: rows streamed from L2 need more than C64_T)
  cudaError_t e = cudaErrorCooperativeLaunchTooLarge;
  for (int ctas = device_sms(); ctas >= 4 && no_room(e); ctas /= 2) {
    (void)cudaGetLastError();
    smem = plan(P, true, std::min(ctas, n), &A);
    const int G = (n + A.R - 1) / A.R;
    e = csr ? run_grid<true>(A, G, smem, st) : run_grid<false>(A, G, smem, st);
  }
  ILM_CHECK_CUDA(e);
  return ILM_OK;
}

}  // namespace ilm
