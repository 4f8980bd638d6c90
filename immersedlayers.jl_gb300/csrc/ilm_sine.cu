// FP64 unbounded-domain inverse Laplacian by sine transforms and discrete
// potential theory (R. A. James, The solution of Poisson's equation for isolated
// source distributions, 1977): the same linear convolution with the lattice Green's
// function G as the zero-padded FFTs of ilm_fft.cu, in a third of the FP64
// operations.
//
// GB300 issues 1.7 FP64 operations per clock and SM, and a zero-padded
// convolution of an n x n field transforms 2n x 2n values both ways: its time
// is its FP64 operation count (2047^2: ~1.0e9 instructions, 2.5 ms).  Here
// the field is never padded in y and transformed in x only:
//
//  1. u1 solves L u1 = f on the box {1..N-1} x {0..n2-1} (N-1 >= n1, f zero in
//     the added columns) with u1 = 0 on the ring of nodes around it: a sine
//     transform of every row (k_sine_rows), then for every mode k the
//     tridiagonal system u_{j+1} + u_{j-1} - 2 cosh(s_k) u_j = F_j,
//     cosh(s_k) = 2 - cos(pi k / N), by its Green's function
//     -a^|j| / (2 sinh s), a = e^-s: one recurrence up, one down (k_modes).
//  2. Extended by zero, u1 satisfies L u1 = f + sigma on the whole lattice with
//     sigma on the ring only (the value of u1 at the neighbouring box node,
//     k_ring_sources); so u1 = G * (f + sigma), and on the ring, where u1 = 0,
//     (G * f) = b := -(G * sigma) (k_ring_potential, (2N + 2 n2)^2 products).
//  3. G * f solves L u = f with u = b on the ring: the mode systems again with
//     b as boundary data, added to u1 (k_modes), and one inverse sine
//     transform (k_sine_rows).
//
// Every step is exact in exact arithmetic; there is no cancellation beyond
// that of the field itself while the box is not much wider than high
// (sine_supported).  Measured against the zero-padded FFTs, us per call:
// 105^2 36 (100), 205^2 51 (155), 405^2 91 (190), 900 x 606 178 (450), 2047^2
// 811 (2450), of which the two sine transforms 440, the modes 200, the ring
// 185; errors against 64-bit references are those of the FFTs (1e-15).
#include <math.h>

#include <algorithm>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "ilm_fftcore.cuh"

namespace ilm {

namespace {

constexpr int SM_T = 256;                  // threads of k_modes
constexpr int SM_WARPS = SM_T / 32;
constexpr int SM_MAX_SMEM = 220 * 1024;

// modes per CTA (consecutive in memory: 4 doubles are one 32-byte sector)
// and chunks of rows per mode
__host__ __device__ constexpr int chunks(int MB) { return SM_T / MB; }
constexpr int SM_LR = 32;                  // most rows of a chunk (a thread's registers)

int modes_per_cta(int n2) { return n2 <= chunks(4) * SM_LR ? 4 : 2; }

// per-mode constants, arrays of N each (mode 0 holds zeros: no such mode)
enum { TB_A = 0, TB_AL, TB_C, TB_IC, TB_D, TB_Q, TB_LAST, TB_P1, TB_HEAD };
// then, per chunk ch: a^(ch L) [chunks], a^(n2 - (ch + 1) L) [chunks]

__global__ void k_mode_table(int N, int n2, int nch, int L, double* __restrict__ tab, double* __restrict__ s2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < 2 * N) s2[k] = k == 0 || k == N ? 0.0 : 2.0 * sinpi((double)k / (double)N);
  if (k >= N) return;
  if (k == 0) {
    for (int q = 0; q < TB_HEAD + 2 * nch; ++q) tab[(size_t)q * N] = 0.0;
    return;
  }
  const double sh = sinpi(0.5 * (double)k / (double)N);
  const double u = 2.0 * sh * sh;              // cosh s - 1
  const double sn = sqrt(u * (u + 2.0));       // sinh s
  const double s = log1p(u + sn);
  const double b = -expm1(-s), a = 1.0 - b;
  tab[(size_t)TB_A * N + k] = a;
  tab[(size_t)TB_AL * N + k] = (1.0 - a) - b;  // a + this = e^-s beyond 64 bits for small s
  tab[(size_t)TB_C * N + k] = 0.5 / sn;
  tab[(size_t)TB_IC * N + k] = -2.0 * sn;
  tab[(size_t)TB_D * N + k] = -1.0 / expm1(-2.0 * s * (n2 + 1.0));
  tab[(size_t)TB_Q * N + k] = exp(-s * (n2 + 1.0));
  tab[(size_t)TB_LAST * N + k] = exp(-s * (double)(n2 - ((n2 - 1) / L) * L));
  tab[(size_t)TB_P1 * N + k] = exp(-s * (double)L);
  for (int ch = 0; ch < nch; ++ch) {
    tab[(size_t)(TB_HEAD + ch) * N + k] = exp(-s * ((double)ch * L));
    tab[(size_t)(TB_HEAD + nch + ch) * N + k] = exp(-s * fmax((double)n2 - (ch + 1.0) * L, 0.0));
  }
}

// Sine transform of rows: f_j, j = 1 .. N-1, from in[row * ldin + j - jin] (zero
// outside [0, nin)), to out[row * ldout + k - kout] = scale * 2 sum_j f_j
// sin(pi j k / N) for k = kout .. kout + nout - 1.  One CTA per pair of rows,
// held as one complex sequence z.
//
// The odd extension of z has the DFT X_k = -2i sum_j z_j sin(pi j k / N).  Its odd
// k are one complex transform of length N / 2: X_{4r+1} = sum_j s_j
// e^{-2 pi i j r / (N/2)} with s_j = e^{-i pi j / N} (p_j - i p_{N/2-j}), p_j = z_j
// + z_{N-j} (k = 3 mod 4 are the r with 4r + 1 > N, X_{2N-k} = -X_k); its even k
// are the same problem of size N / 2 on z_j - z_{N-j}.  So levels of length
// N/2, N/4, .. make up a pair of rows (N complex points for two rows: the
// optimum of a real transform, without the split and the running sum of the
// usual real algorithm, whose rounding errors grow along the row).  All levels
// advance together, one radix-4 / 3 / 2 Stockham stage at a time.
//
// FP64-issue bound from N ~ 512 (three quarters of the operations are the
// butterflies).  Below, a dependent FP64 operation takes 64 clocks whatever the
// number of active lanes, so SPLIT gives every real output of a radix-2 (or 3)
// stage its own thread: two (four) FMAs deep instead of a 28-operation
// radix-4 butterfly per thread.
struct Radix {
  int r, Ns;  // r = 1: done
};
// stage s of a transform of 2^x 3^y points (y <= 1): 4s, then 3, then 2
__device__ __forceinline__ Radix stage_radix(int x, int y, int s) {
  const int h = x >> 1;
  if (s < h) return Radix{4, 1 << (2 * s)};
  if (y && s == h) return Radix{3, 1 << (2 * h)};
  if ((x & 1) && s == h + y) return Radix{2, (y ? 3 : 1) << (2 * h)};
  return Radix{1, 0};
}
constexpr int SR_T = 256;        // threads of k_sine_rows
constexpr int SR_SPLIT_N = 256;  // largest N of the split stages (two outputs per thread)
constexpr int SR_FOLD_N = 1024;  // largest N of the split folds

template <bool SPLIT, bool FOLD>
__global__ void __launch_bounds__(SR_T) k_sine_rows(int N, int lx, int ly, int nrows, const double* __restrict__ in,
                                                    int ldin, int nin, int jin, double* __restrict__ out, int ldout,
                                                    int nout, int kout, double scale, const double2* __restrict__ tw) {
  // N = 2^lx 3^ly; level l: length N >> (l + 1), at offset N - (N >> l)
  extern __shared__ __align__(16) double2 sm2[];
  const int t = threadIdx.x;
  double2* A = sm2;
  double2* B = A + N;
  double* z = reinterpret_cast<double*>(B);  // z[2 j + component]
  const int row = 2 * blockIdx.x;
  const bool two = row + 1 < nrows;
  const double* __restrict__ xa = in + (size_t)row * ldin - jin;
  const double* __restrict__ xb = xa + ldin;
  pdl_wait();
  unsigned any = 0u;
  for (int j = t; j < N; j += SR_T) {
    const bool ok = j >= 1 && j >= jin && j < jin + nin;
    const double2 v = make_double2(ok ? xa[j] : 0.0, ok && two ? xb[j] : 0.0);
    any |= (unsigned)__double2hiint(v.x) << 1 | (unsigned)__double2loint(v.x) | (unsigned)__double2hiint(v.y) << 1 |
           (unsigned)__double2loint(v.y);
    B[j] = v;
  }
  // rows of zeros (beyond the bodies, where a source is regularized surface
  // data): no transform
  if (!__syncthreads_or(any != 0u)) {
    for (int i = t; i < nout; i += SR_T) {
      out[(size_t)row * ldout + i] = 0.0;
      if (two) out[(size_t)(row + 1) * ldout + i] = 0.0;
    }
    return;
  }
  if (FOLD) {
    // folds: level l leaves p_j at N_l - j and hands z_j - z_{N_l - j} at j to the next
    for (int l = 0; l < lx; ++l) {
      const int Nl = N >> l, H = Nl >> 1;
      for (int i = t; i < 2 * (H - 1); i += SR_T) {
        const int lo = i + 2, hi = 2 * (Nl - (lo >> 1)) + (lo & 1);
        const double u = z[lo], v = z[hi];
        z[lo] = u - v;
        z[hi] = u + v;
      }
      if (Nl > 32) __syncthreads();  // below, 2 (H - 1) < 32 items: one warp
      else __syncwarp();
    }
    __syncthreads();
    // s_j of every level
    for (int i = t; i < 2 * N; i += SR_T) {
      const int o = i >> 1;
      int l = 0;
      while ((N >> (l + 1)) >= N - o) ++l;
      if (l >= lx) continue;
      const int Nl = N >> l, H = Nl >> 1, j = o - (N - Nl);
      const double2 w = tw[j << l];
      double2 g;  // p_j - i p_{H-j}
      if (j == 0) {
        const double2 h = B[H];
        g = make_double2(2.0 * h.y, -2.0 * h.x);
      } else {
        const double2 p = B[Nl - j], h = B[H + j];
        g = make_double2(p.x + h.y, p.y - h.x);
      }
      if (i & 1) A[o].y = fma(w.x, g.y, w.y * g.x);
      else A[o].x = fma(w.x, g.x, -(w.y * g.y));
    }
  } else {
    // folds and s_j together: j, H - j, H + j and N_l - j are a closed set
    for (int l = 0; l < lx; ++l) {
      const int Nl = N >> l, H = Nl >> 1;
      double2* S = A + (N - Nl);
      for (int j = t; 2 * j <= H; j += SR_T) {
        const double2 z1 = B[H + j], z0 = B[H - j];  // j = 0: both z_H
        if (j == 0) {
          S[0] = make_double2(2.0 * z0.y, -2.0 * z0.x);
          continue;
        }
        const double2 y0 = B[j], y1 = B[Nl - j];
        const double2 pj = cadd(y0, y1), mj = csub(y0, y1), ph = cadd(z0, z1), mh = csub(z0, z1);
        S[j] = cmul(tw[j << l], make_double2(pj.x + ph.y, pj.y - ph.x));
        B[j] = mj;
        if (2 * j < H) {
          S[H - j] = cmul(tw[(H - j) << l], make_double2(ph.x + pj.y, ph.y - pj.x));
          B[H - j] = mh;
        }
      }
      if (Nl > 64) __syncthreads();  // below, one warp
      else __syncwarp();
    }
    __syncthreads();
  }
  // what is left of N = 3 * 2^lx: two values
  double2 tail1 = make_double2(0.0, 0.0), tail2 = tail1;
  if (ly) {
    const double q = 1.7320508075688772935;
    const double2 z1 = B[1], z2 = B[2];
    tail1 = make_double2(q * (z1.x + z2.x), q * (z1.y + z2.y));
    tail2 = make_double2(q * (z1.x - z2.x), q * (z1.y - z2.y));
  }
  __syncthreads();
  // Stockham stages of all levels; a level that is done stays where its last
  // stage left it (B after an odd number)
  if (SPLIT) {
    for (int st = 0; st < lx - 1 + ly; ++st) {
      const double2* a = (st & 1) ? B : A;
      double* b = reinterpret_cast<double*>((st & 1) ? A : B);
      for (int i = t; i < 2 * N; i += SR_T) {
        const int o = i >> 1;
        int l = 0;
        while ((N >> (l + 1)) >= N - o) ++l;
        const int x = lx - 1 - l, off = N - (N >> l), k = o - off, len = N >> (l + 1);
        if (x < 0 || k >= len || st >= x + ly) continue;
        const double2* y = a + off;
        if (st < x) {
          const int Ns = 1 << st, q = k & (Ns - 1), m = (k >> st) & 1, j = ((k >> (st + 1)) << st) + q;
          const double2 w = tw[q * (N >> st) + m * N], v = y[j + (len >> 1)];
          const double a0 = (i & 1) ? y[j].y : y[j].x;
          b[i] = (i & 1) ? fma(w.x, v.y, fma(w.y, v.x, a0)) : fma(w.x, v.x, fma(-w.y, v.y, a0));
        } else {
          const int Ns = 1 << x, m = k >> x, q = k & (Ns - 1), M = 2 * N, e = q * (M / (3 * Ns)) + m * (M / 3);
          const double2 w1 = tw[e % M], w2 = tw[2 * e % M], v1 = y[q + Ns], v2 = y[q + 2 * Ns];
          double r = (i & 1) ? y[q].y : y[q].x;
          if (i & 1) r = fma(w1.x, v1.y, fma(w1.y, v1.x, fma(w2.x, v2.y, fma(w2.y, v2.x, r))));
          else r = fma(w1.x, v1.x, fma(-w1.y, v1.y, fma(w2.x, v2.x, fma(-w2.y, v2.y, r))));
          b[i] = r;
        }
      }
      __syncthreads();
    }
  } else {
    const int stages = ((lx - 1) >> 1) + ((lx - 1) & 1) + ly;  // of the longest level: no level has more
    const double s3 = 0.86602540378443864676;
    for (int st = 0; st < stages; ++st) {
      const double2* a = (st & 1) ? B : A;
      double2* b = (st & 1) ? A : B;
      for (int idx = t;; idx += SR_T) {
        int j = idx, l = 0;
        Radix R{1, 0};
        for (; l < lx; ++l) {
          R = stage_radix(lx - 1 - l, ly, st);
          const int cnt = R.r == 1 ? 0 : R.r == 4 ? N >> (l + 3) : (N >> (l + 1)) / R.r;
          if (j < cnt) break;
          j -= cnt;
        }
        if (l == lx) break;
        const int len = N >> (l + 1), stride = R.r == 4 ? len >> 2 : len / R.r, off = N - (N >> l);
        const double2* x = a + off;
        double2* y = b + off;
        const int q = R.r == 3 || R.Ns % 3 != 0 ? j & (R.Ns - 1) : j % R.Ns;
        const int step = q * ((2 * N) / (R.Ns * R.r));
        const int base = (j - q) * R.r + q;
        double2 a0 = x[j], a1 = x[j + stride];
        if (R.r == 4) {
          double2 a2 = x[j + 2 * stride], a3 = x[j + 3 * stride];
          if (q != 0) {
            a1 = cmul(a1, tw[step]);
            a2 = cmul(a2, tw[2 * step]);
            a3 = cmul(a3, tw[3 * step]);
          }
          const double2 s02 = cadd(a0, a2), d02 = csub(a0, a2), s13 = cadd(a1, a3), d13 = csub(a1, a3);
          y[base] = cadd(s02, s13);
          y[base + R.Ns] = make_double2(d02.x + d13.y, d02.y - d13.x);
          y[base + 2 * R.Ns] = csub(s02, s13);
          y[base + 3 * R.Ns] = make_double2(d02.x - d13.y, d02.y + d13.x);
        } else if (R.r == 3) {
          double2 a2 = x[j + 2 * stride];
          if (q != 0) {
            a1 = cmul(a1, tw[step]);
            a2 = cmul(a2, tw[2 * step]);
          }
          const double2 s12 = cadd(a1, a2), d12 = csub(a1, a2);
          const double mx = fma(-0.5, s12.x, a0.x), my = fma(-0.5, s12.y, a0.y);
          y[base] = cadd(a0, s12);
          y[base + R.Ns] = make_double2(fma(s3, d12.y, mx), fma(-s3, d12.x, my));
          y[base + 2 * R.Ns] = make_double2(fma(-s3, d12.y, mx), fma(s3, d12.x, my));
        } else {
          if (q != 0) a1 = cmul(a1, tw[step]);
          y[base] = cadd(a0, a1);
          y[base + R.Ns] = csub(a0, a1);
        }
      }
      __syncthreads();
    }
  }
  // X_k -> 2 sum f sin: rows are -Im and Re
  double* __restrict__ oa = out + (size_t)row * ldout;
  double* __restrict__ ob = oa + ldout;
  for (int i = t; i < nout; i += SR_T) {
    const int k = i + kout;
    double2 v = make_double2(0.0, 0.0);
    if (k > 0) {
      const int l = __ffs(k) - 1;
      if (l >= lx) {
        v = (k >> lx) == 1 ? tail1 : tail2;
      } else {
        const int Nl = N >> l, kl = k >> l;
        const bool neg = (kl & 3) == 3;
        const int r = neg ? (2 * Nl - kl - 1) >> 2 : (kl - 1) >> 2;
        const int x = lx - 1 - l, ns = SPLIT ? x + ly : (x >> 1) + (x & 1) + ly;
        const double2 X = ((ns & 1) ? B : A)[N - Nl + r];
        v = neg ? make_double2(X.y, -X.x) : make_double2(-X.y, X.x);
      }
    }
    oa[i] = scale * v.x;
    if (two) ob[i] = scale * v.y;
  }
}

// sum over the chunks of one mode, in every thread of the mode
template <int MB>
__device__ __forceinline__ double mode_sum(double v, double* red) {
  const int t = threadIdx.x, m = t % MB;
#pragma unroll
  for (int o = 16; o >= MB; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((t & 31) < MB) red[(t >> 5) * MB + m] = v;
  __syncthreads();
  // lane (w, m) takes warp w's sum (lanes beyond the warps: none)
  double s = (t & 31) < SM_WARPS * MB ? red[t & 31] : 0.0;
#pragma unroll
  for (int o = 16; o >= MB; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __syncthreads();
  return s;
}

// The tridiagonal systems of MB modes: U (n2 rows of N modes, the mode index
// fastest) holds the right-hand sides and receives the solutions with zero
// boundary values (SECOND = false), or U += the solution for the ring's
// boundary data (SECOND = true).  All values carry the factor 2 of
// k_sine_rows.
//
// A mode's rows are cut into chunks(MB) chunks of L <= LR, one thread each, and
// stay in its registers.  Pass 1 runs v_j = F_j + a v_{j-1} and y_j = F_j +
// a y_{j+1} from zero over every chunk; the results are combined into each
// chunk's starting values (shuffles within a warp, one warp across warps);
// pass 2 forms v from those, and from u = -c (v_j + a y_{j+1}) at the chunk's
// last row goes down by u_j = a (u_{j+1} - v_j).  The homogeneous solutions
// that meet the boundary values obey the same recurrences, so they enter as
// starting values.  Five FP64 instructions per value, which bound the kernel.
//
// The lowest eighth of the modes take a in two parts (FINE): a's rounding
// error, repeated over the ~1/s rows that a value reaches, would show as
// eps / s.
template <int MB, int LR, bool SECOND, bool FINE>
__device__ __forceinline__ void modes_body(int N, int n2, int L, double* __restrict__ U,
                                           const double* __restrict__ tab, const double* __restrict__ s2,
                                           const double* __restrict__ bsum, const double* __restrict__ bdif,
                                           const double* __restrict__ bbot, const double* __restrict__ btop) {
  constexpr int NCH = chunks(MB), CW = 32 / MB;  // chunks, chunks per warp
  __shared__ double red[SM_WARPS * MB], wv[SM_WARPS * MB], wy[SM_WARPS * MB], tv[2 * MB];
  const int t = threadIdx.x, m = t % MB, ch = t / MB, lane = t & 31, warp = t >> 5;
  const int k = blockIdx.x * MB + m;
  const int j0 = min(ch * L, n2), nj = min(L, n2 - j0), chl = (n2 - 1) / L;
  const double a = tab[(size_t)TB_A * N + k], al = FINE ? tab[(size_t)TB_AL * N + k] : 0.0;
  const double c = tab[(size_t)TB_C * N + k], ic = tab[(size_t)TB_IC * N + k];
  const double dq = tab[(size_t)TB_D * N + k], q = tab[(size_t)TB_Q * N + k];
  const double head = tab[(size_t)(TB_HEAD + ch) * N + k], tail = tab[(size_t)(TB_HEAD + NCH + ch) * N + k];
  const double last = tab[(size_t)TB_LAST * N + k];
  // a x + f
  auto step = [&](double x, double f) { return FINE ? fma(a, x, fma(al, x, f)) : fma(a, x, f); };
  double F[LR];
  double g0 = 0.0, g1 = 0.0;
  double* __restrict__ u0 = U + (size_t)j0 * N + k;
  pdl_wait();
  if (SECOND) {
    // sine transforms of the ring's bottom and top values (modes of this CTA)
    double b0 = 0.0, b1 = 0.0;
    const int M = 2 * N, dx = (k * NCH) % M;
    int at = (k * (1 + ch)) % M;
    for (int i = 1 + ch; i < N; i += NCH) {
      const double s = s2[at];
      b0 = fma(bbot[i], s, b0);
      b1 = fma(btop[i], s, b1);
      at += dx;
      if (at >= M) at -= M;
    }
    g0 = mode_sum<MB>(b0, red);
    g1 = mode_sum<MB>(b1, red);
    const double* __restrict__ e = (k & 1) ? bsum : bdif;
    const double sc = -s2[k];
#pragma unroll
    for (int i = 0; i < LR; ++i) F[i] = i < nj ? sc * e[j0 + i] : 0.0;
  } else {
#pragma unroll
    for (int i = 0; i < LR; ++i) F[i] = i < nj ? u0[(size_t)i * N] : 0.0;
  }
  double v = 0.0, y = 0.0;
#pragma unroll
  for (int i = 0; i < LR; ++i) {
    if (i < nj) v = step(v, F[i]);
    if (LR - 1 - i < nj) y = step(y, F[LR - 1 - i]);
  }
  // v of the last row (its chunk may be short), before the carries
  if (ch == chl) tv[m] = v;
  // inclusive scans over the warp's chunks: v upwards, y downwards (past the
  // last rows both are zero)
  double iv = v, iy = y, P = tab[(size_t)TB_P1 * N + k];
#pragma unroll
  for (int o = 1; o < CW; o <<= 1) {
    const double pv = __shfl_up_sync(0xffffffffu, iv, o * MB), py = __shfl_down_sync(0xffffffffu, iy, o * MB);
    if (lane >= o * MB) iv = fma(P, pv, iv);
    if (lane + o * MB < 32) iy = fma(P, py, iy);
    P *= P;  // a^(o L); after the last round a^(CW L)
  }
  if (lane >= 32 - MB) wv[warp * MB + m] = iv;
  if (lane < MB) wy[warp * MB + m] = iy;
  double v0 = __shfl_up_sync(0xffffffffu, iv, MB), y0 = __shfl_down_sync(0xffffffffu, iy, MB);
  if (lane < MB) v0 = 0.0;
  if (lane >= 32 - MB) y0 = 0.0;
  __syncthreads();
  if (warp == 0 && lane < 2 * MB) {  // carries into every warp: v lanes [0, MB), y lanes [MB, 2 MB)
    const bool up = lane < MB;
    double* w = up ? wv : wy;
    double carry = 0.0;
    for (int s = 0; s < SM_WARPS; ++s) {
      const int at = (up ? s : SM_WARPS - 1 - s) * MB + m;
      const double x = w[at];
      w[at] = carry;
      carry = fma(P, carry, x);
    }
    if (!up) tv[MB + m] = carry;  // y of row 0
  }
  __syncthreads();
  // starting values without the boundary terms: the warp's carry, over the
  // chunks of the warp between
  v0 = fma(tab[(size_t)(TB_HEAD + (ch % CW)) * N + k], wv[warp * MB + m], v0);
  y0 = fma(tab[(size_t)(TB_HEAD + (CW - 1 - ch % CW)) * N + k], wy[warp * MB + m], y0);
  if (ch == chl) tv[m] = fma(last, v0, tv[m]);  // v of row n2 - 1
  __syncthreads();
  const double vl = tv[m], yf = tv[MB + m];
  {  // boundary terms: u_{-1} = g0, u_{n2} = g1
    const double ca = c * a;
    const double Ab = fma(ca, yf, g0), Bb = fma(ca, vl, g1);
    v0 = fma(head, (Ab - q * Bb) * dq * ic, v0);
    const double yb = (Bb - q * Ab) * dq * ic;
    y0 = j0 + nj < n2 ? fma(tail, yb, y0) : yb;
  }
#pragma unroll
  for (int i = 0; i < LR; ++i)
    if (i < nj) F[i] = v0 = step(v0, F[i]);
  const double ul = -c * step(y0, v0);  // at the chunk's last row
  double u = ul;
#pragma unroll
  for (int i = LR - 1; i >= 0; --i) {
    if (i < nj) {
      const double d = u - F[i], w = FINE ? fma(a, d, al * d) : a * d;
      u = i == nj - 1 ? ul : w;
      F[i] = u;
    }
  }
  // The rows beside the ring are its sources, and there -c (v + a y) is the
  // small difference of large numbers: a sum of the products with
  // sinh((n2 - j) s) / sinh((n2 + 1) s) instead.
  const double ub = -a * (yf - q * vl) * dq, ut = -a * (vl - q * yf) * dq;
#pragma unroll
  for (int i = 0; i < LR; ++i)
    if (i < nj) {
      double* o = u0 + (size_t)i * N;
      if (SECOND) *o += F[i];
      else *o = j0 + i == 0 ? ub : j0 + i == n2 - 1 ? ut : F[i];
    }
}

template <int MB, int LR, bool SECOND>
__global__ void __launch_bounds__(SM_T, 2) k_modes(int N, int n2, int L, double* __restrict__ U,
                                                const double* __restrict__ tab, const double* __restrict__ s2,
                                                const double* __restrict__ bsum, const double* __restrict__ bdif,
                                                const double* __restrict__ bbot, const double* __restrict__ btop) {
  if ((int)blockIdx.x * MB < N / 8)
    modes_body<MB, LR, SECOND, true>(N, n2, L, U, tab, s2, bsum, bdif, bbot, btop);
  else
    modes_body<MB, LR, SECOND, false>(N, n2, L, U, tab, s2, bsum, bdif, bbot, btop);
}

// Sources on the ring from the modes of u1 (one warp each): u1 beside the left
// and right ends of row j, and u1 in the bottom and top rows at column i.
__global__ void __launch_bounds__(256) k_ring_sources(int N, int n2, const double* __restrict__ U,
                                                      const double* __restrict__ s2, double* __restrict__ Sb,
                                                      double* __restrict__ St, double* __restrict__ Sl,
                                                      double* __restrict__ Sr) {
  const int id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  if (id >= n2 + N) return;
  const double f = 0.5 / (double)N;  // (2 / N), the factor 2 and the table's 2 sin
  double a0 = 0.0, a1 = 0.0;
  if (id < n2) {
    const double* u = U + (size_t)id * N;
    for (int k = lane; k < N; k += 64) {
      a0 = fma(s2[k], u[k], a0);
      if (k + 32 < N) a1 = fma(s2[k + 32], u[k + 32], a1);
    }
    a0 += a1;
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    const double other = __shfl_xor_sync(0xffffffffu, a0, 1);  // lane 0: even modes, lane 1: odd
    if (lane == 0) {
      Sl[id] = f * (other + a0);
      Sr[id] = f * (other - a0);
    }
    return;
  }
  const int i = id - n2, M = 2 * N, dx = (32 * i) % M;
  const double* ub = U;
  const double* ut = U + (size_t)(n2 - 1) * N;
  int at = (lane * i) % M;
  for (int k = lane; k < N; k += 32) {
    const double s = s2[at];
    a0 = fma(s, ub[k], a0);
    a1 = fma(s, ut[k], a1);
    at += dx;
    if (at >= M) at -= M;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
  }
  if (lane == 0) {
    Sb[i] = i == 0 ? 0.0 : f * a0;
    St[i] = i == 0 ? 0.0 : f * a1;
  }
}

// Ring potentials b = -(G * sigma), one warp per pair of opposite targets:
// bottom and top at column i (1 .. N-1), left and right at row j.  T: G(m, n),
// row stride ld, symmetric.  FP64-issue bound: 4 (N + n2) FMAs per pair.
__global__ void __launch_bounds__(256) k_ring_potential(int N, int n2, const double* __restrict__ T, int ld,
                                                        const double* __restrict__ Sb, const double* __restrict__ St,
                                                        const double* __restrict__ Sl, const double* __restrict__ Sr,
                                                        double* __restrict__ bbot, double* __restrict__ btop,
                                                        double* __restrict__ bsum, double* __restrict__ bdif) {
  const int id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  if (id >= n2 + N) return;
  double p0 = 0.0, p1 = 0.0, r0 = 0.0, r1 = 0.0;
  if (id < n2) {
    const int j = id;
    const double* h1 = T + (size_t)N * ld;
    const double* ga = T + (size_t)(j + 1) * ld;
    const double* gb = T + (size_t)(n2 - j) * ld;
    for (int s = lane; s < n2; s += 32) {
      const double h = T[abs(j - s)], g = h1[abs(j - s)], l = Sl[s], r = Sr[s];
      p0 = fma(h, l, p0);
      r0 = fma(g, l, r0);
      p1 = fma(g, r, p1);
      r1 = fma(h, r, r1);
    }
    for (int s = 1 + lane; s < N; s += 32) {
      const double A = ga[s], B = gb[s];
      p0 = fma(A, Sb[s], p0);
      p1 = fma(B, St[s], p1);
      r0 = fma(A, Sb[N - s], r0);
      r1 = fma(B, St[N - s], r1);
    }
  } else {
    const int i = id - n2;
    const double* h1 = T + (size_t)(n2 + 1) * ld;
    const double* ga = T + (size_t)i * ld;
    const double* gb = T + (size_t)(N - i) * ld;
    for (int s = 1 + lane; s < N; s += 32) {
      const double h = T[abs(i - s)], g = h1[abs(i - s)], b = Sb[s], u = St[s];
      p0 = fma(h, b, p0);
      r0 = fma(g, b, r0);
      p1 = fma(g, u, p1);
      r1 = fma(h, u, r1);
    }
    for (int s = lane; s < n2; s += 32) {
      const double A = ga[s + 1], B = gb[s + 1];
      p0 = fma(A, Sl[s], p0);
      p1 = fma(B, Sr[s], p1);
      r0 = fma(A, Sl[n2 - 1 - s], r0);
      r1 = fma(B, Sr[n2 - 1 - s], r1);
    }
  }
  p0 += p1;
  r0 += r1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    p0 += __shfl_xor_sync(0xffffffffu, p0, o);
    r0 += __shfl_xor_sync(0xffffffffu, r0, o);
  }
  if (lane == 0) {
    if (id < n2) {
      bsum[id] = -(p0 + r0);
      bdif[id] = r0 - p0;
    } else {
      bbot[id - n2] = -p0;
      btop[id - n2] = -r0;
    }
  }
}

__global__ void k_copy_table(const double* __restrict__ src, int lds, int n, double* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[(size_t)blockIdx.y * n + i] = src[(size_t)blockIdx.y * lds + i];
}

// The tables in use -- mode tables by (N, n2), copies of G by size -- and the last
// few beside them (a cache that is made again finds its own): kKeptBytes at most.
// (G is copied because the library's table, as large as its largest user, spreads a
// small one's rows over its long ones: 0.7 us of 48 at 105^2.)
using TabKey = std::tuple<int, int, int>;
enum { TAB_MODES, TAB_LGF };
constexpr size_t kKeptBytes = 64 << 20;
struct TableCache {
  std::mutex mu;
  std::map<TabKey, std::weak_ptr<const double>> all;
  std::deque<std::pair<DevTable, size_t>> kept;
  size_t bytes = 0;
};
TableCache& table_cache() {
  static TableCache* p = new TableCache;  // (not destroyed: the driver may be gone by then)
  return *p;
}
DevTable find_table(const TabKey& key) {
  TableCache& T = table_cache();
  std::lock_guard<std::mutex> lk(T.mu);
  auto it = T.all.find(key);
  return it == T.all.end() ? nullptr : it->second.lock();
}
// the first one added wins
DevTable add_table(const TabKey& key, const DevTable& t, size_t bytes) {
  TableCache& T = table_cache();
  std::vector<DevTable> old;  // (freed after the lock)
  std::lock_guard<std::mutex> lk(T.mu);
  for (auto it = T.all.begin(); it != T.all.end();) it = it->second.expired() ? T.all.erase(it) : std::next(it);
  auto it = T.all.find(key);
  if (it != T.all.end())
    if (DevTable first = it->second.lock()) return first;
  T.all[key] = t;
  T.kept.emplace_back(t, bytes);
  T.bytes += bytes;
  while (T.bytes > kKeptBytes) {
    old.push_back(T.kept.front().first);
    T.bytes -= T.kept.front().second;
    T.kept.pop_front();
  }
  return t;
}
int new_table(size_t bytes, double** d, DevTable* t) {
  if (cudaMalloc(d, bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    set_error("cudaMalloc of a sine-transform table (%zu bytes) failed", bytes);
    return ILM_ERR_NO_MEMORY;
  }
  *t = dev_table(*d);
  return ILM_OK;
}

}  // namespace

// The box {1..N-1} must not be much wider than high: the boundary terms
// divide by 1 - a^(2 (n2 + 1)), which for the lowest mode (s ~ pi / N) loses
// N / (2 pi n2) in relative accuracy.
bool sine_supported(int n1, int n2) {
  const int N = good_fft_size(n1 + 1);
  return n2 >= 4 && 8 * n2 >= N && n2 <= chunks(2) * SM_LR;
}

int sine_plan_init(SinePlan* p, int n1, int n2, const void* tw, cudaStream_t st) {
  p->n1 = n1;
  p->n2 = n2;
  const int N = p->N = good_fft_size(n1 + 1);
  p->tw = tw;
  p->MB = modes_per_cta(n2);
  const int nch = chunks(p->MB);
  p->L = (n2 + nch - 1) / nch;
  const size_t ntab = (size_t)(TB_HEAD + 2 * nch) * N;
  const TabKey modes(TAB_MODES, N, n2);
  p->tab_own = find_table(modes);
  if (!p->tab_own) {
    const size_t bytes = (ntab + 2 * (size_t)N) * sizeof(double);
    double* d = nullptr;
    DevTable t;
    ILM_TRY(new_table(bytes, &d, &t));
    k_mode_table<<<(2 * N + 127) / 128, 128, 0, st>>>(N, n2, nch, p->L, d, d + ntab);
    ILM_CHECK_LAUNCH();
    ILM_CHECK_CUDA(cudaStreamSynchronize(st));
    p->tab_own = add_table(modes, t, bytes);
  }
  p->tab = p->tab_own.get();
  p->s2 = p->tab + ntab;
  const int M = std::max(N, n2 + 1);
  const TabKey lgf(TAB_LGF, M, 0);
  p->ldg = M + 1;
  p->lgf_own = find_table(lgf);
  if (!p->lgf_own) {
    const size_t bytes = (size_t)(M + 1) * (M + 1) * sizeof(double);
    double* d = nullptr;
    DevTable t, G;  // (G stays while it is copied)
    int ld = 0;
    ILM_TRY(lgf_table_shared(M, &G, &ld, st));
    ILM_TRY(new_table(bytes, &d, &t));
    k_copy_table<<<dim3((M + 1 + 255) / 256, M + 1), 256, 0, st>>>(G.get(), ld, M + 1, d);
    ILM_CHECK_LAUNCH();
    ILM_CHECK_CUDA(cudaStreamSynchronize(st));
    p->lgf_own = add_table(lgf, t, bytes);
  }
  p->lgf = p->lgf_own.get();
  return p->work.alloc(((size_t)n2 * N + 4 * (size_t)N + 4 * (size_t)n2) * sizeof(double));
}

int sine_apply(SinePlan* p, const double* in, double* out, double inv_factor, cudaStream_t st) {
  const int n1 = p->n1, n2 = p->n2, N = p->N;
  double* U = p->work.as<double>();
  double *Sb = U + (size_t)n2 * N, *St = Sb + N, *bb = St + N, *bt = bb + N;
  double *Sl = bt + N, *Sr = Sl + n2, *bs = Sr + n2, *bd = bs + n2;
  const double2* tw = static_cast<const double2*>(p->tw);
  int lx = 0;
  while (((N >> lx) & 1) == 0) ++lx;
  const int ly = (N >> lx) == 3 ? 1 : 0;
  const size_t smr = 2 * (size_t)N * sizeof(double2);
  const int rb = (n2 + N + 7) / 8;
  auto rows = N <= SR_SPLIT_N ? k_sine_rows<true, true> : N <= SR_FOLD_N ? k_sine_rows<false, true> : k_sine_rows<false, false>;
  ILM_CHECK_CUDA(cudaFuncSetAttribute(rows, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_MAX_SMEM));
  auto modes = [&](bool second) -> int {
    using K = void (*)(int, int, int, double*, const double*, const double*, const double*, const double*,
                       const double*, const double*);
    static const K table[2][6] = {
        {k_modes<4, 1, false>, k_modes<4, 2, false>, k_modes<4, 4, false>, k_modes<4, 8, false>,
         k_modes<4, 16, false>, k_modes<4, 32, false>},
        {k_modes<4, 1, true>, k_modes<4, 2, true>, k_modes<4, 4, true>, k_modes<4, 8, true>, k_modes<4, 16, true>,
         k_modes<4, 32, true>}};
    int r = 0;
    while ((1 << r) < p->L) ++r;
    const K k = p->MB == 4 ? table[second][r] : second ? k_modes<2, 32, true> : k_modes<2, 32, false>;
    ILM_CHECK_CUDA(launch_pdl(k, dim3(N / p->MB), dim3(SM_T), st, N, n2, p->L, U, p->tab, p->s2, bs, bd, bb, bt));
    return ILM_OK;
  };
  ILM_CHECK_CUDA(launch_pdl_smem(rows, dim3((n2 + 1) / 2), dim3(SR_T), smr, st, N, lx, ly, n2, in, n1, n1, 1, U,
                                 N, N, 0, 1.0, tw));
  ILM_TRY(modes(false));
  ILM_CHECK_CUDA(launch_pdl_smem(k_ring_sources, dim3(rb), dim3(256), 0, st, N, n2, (const double*)U, p->s2, Sb, St,
                                 Sl, Sr));
  ILM_CHECK_CUDA(launch_pdl_smem(k_ring_potential, dim3(rb), dim3(256), 0, st, N, n2, p->lgf, p->ldg,
                                 (const double*)Sb, (const double*)St, (const double*)Sl, (const double*)Sr, bb, bt,
                                 bs, bd));
  ILM_TRY(modes(true));
  // 2 from each transform, 2 / N of the inverse
  ILM_CHECK_CUDA(launch_pdl_smem(rows, dim3((n2 + 1) / 2), dim3(SR_T), smr, st, N, lx, ly, n2, (const double*)U,
                                 N, N, 0, out, n1, n1, 1, inv_factor / (2.0 * N), tw));
  return ILM_OK;
}

}  // namespace ilm
