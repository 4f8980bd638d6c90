// Complex arithmetic and the shared-memory Stockham transform used by the FFT
// convolution (ilm_fft.cu) and the sine-transform solver (ilm_sine.cu).
#pragma once

#include "ilm_internal.cuh"

namespace ilm {

template <typename T> struct CT;
template <> struct CT<float> { using t = float2; };
template <> struct CT<double> { using t = double2; };

template <typename C> __device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
// s * i * a  (s = +1 or -1)
template <typename C> __device__ __forceinline__ C cmuli(C a, int s) {
  C r; r.x = -s * a.y; r.y = s * a.x; return r;
}

// Stockham auto-sort FFT of `ncol` columns of length L, column c at A[c*cs ..].
// tw: table of length twlen (multiple of L) with tw[m] = exp(-2 pi i m / twlen).
// SIGN = -1 forward, +1 inverse (unnormalised).  Returns the buffer holding
// the result (A or B).  Must be called by all threads of the block.
template <typename T, int SIGN>
__device__ typename CT<T>::t* stockham(typename CT<T>::t* A, typename CT<T>::t* B, int L, int ncol, int cs,
                                      const typename CT<T>::t* __restrict__ tw, int twlen) {
  using C = typename CT<T>::t;
  int Ns = 1;
  int rem = L;
  const T s3 = (T)0.86602540378443864676;
  while (rem > 1) {
    const int r = (rem % 4 == 0) ? 4 : ((rem % 3 == 0) ? 3 : 2);
    const int stride = L / r;
    const int tstep0 = twlen / (Ns * r);
    for (int idx = threadIdx.x; idx < ncol * stride; idx += blockDim.x) {
      const int c = idx / stride;
      const int j = idx - c * stride;
      const C* a_in = A + (size_t)c * cs;
      C* b_out = B + (size_t)c * cs;
      const int k = j % Ns;
      const int tstep = tstep0 * k;
      C a0 = a_in[j];
      C a1 = a_in[j + stride];
      C a2, a3;
      if (r > 2) a2 = a_in[j + 2 * stride];
      if (r > 3) a3 = a_in[j + 3 * stride];
      if (k != 0) {
        C w = tw[tstep];
        if (SIGN > 0) w.y = -w.y;
        a1 = cmul(a1, w);
        if (r > 2) {
          C w2 = tw[2 * tstep];
          if (SIGN > 0) w2.y = -w2.y;
          a2 = cmul(a2, w2);
        }
        if (r > 3) {
          C w3 = tw[3 * tstep];
          if (SIGN > 0) w3.y = -w3.y;
          a3 = cmul(a3, w3);
        }
      }
      const int base = (j / Ns) * Ns * r + k;
      if (r == 2) {
        b_out[base] = cadd(a0, a1);
        b_out[base + Ns] = csub(a0, a1);
      } else if (r == 4) {
        C s02 = cadd(a0, a2), d02 = csub(a0, a2);
        C s13 = cadd(a1, a3), d13 = csub(a1, a3);
        C id = cmuli(d13, SIGN);
        b_out[base] = cadd(s02, s13);
        b_out[base + Ns] = cadd(d02, id);
        b_out[base + 2 * Ns] = csub(s02, s13);
        b_out[base + 3 * Ns] = csub(d02, id);
      } else {  // r == 3
        C s12 = cadd(a1, a2), d12 = csub(a1, a2);
        C m;
        m.x = a0.x - (T)0.5 * s12.x;
        m.y = a0.y - (T)0.5 * s12.y;
        C id = cmuli(d12, SIGN);
        id.x *= s3;
        id.y *= s3;
        b_out[base] = cadd(a0, s12);
        b_out[base + Ns] = cadd(m, id);
        b_out[base + 2 * Ns] = csub(m, id);
      }
    }
    __syncthreads();
    C* t = A;
    A = B;
    B = t;
    Ns *= r;
    rem /= r;
  }
  return A;
}

// ---------------------------------------------------------------------------
// DFTs held in registers (FP32)
// ---------------------------------------------------------------------------
// exp(-2 pi i k / N) for N = 32 and 24 as literals: in the unrolled register
// DFTs k is a compile-time constant, so the switch folds to an immediate and
// the multiplications by the trivial factors (0, +-1, +-1/2) simplify
__device__ __forceinline__ float2 tw32(int k) {
  switch (k) {
    case 0: return make_float2(1.000000000e+00f, 0.000000000e+00f);
    case 1: return make_float2(9.807852804e-01f, -1.950903220e-01f);
    case 2: return make_float2(9.238795325e-01f, -3.826834324e-01f);
    case 3: return make_float2(8.314696123e-01f, -5.555702330e-01f);
    case 4: return make_float2(7.071067812e-01f, -7.071067812e-01f);
    case 5: return make_float2(5.555702330e-01f, -8.314696123e-01f);
    case 6: return make_float2(3.826834324e-01f, -9.238795325e-01f);
    case 7: return make_float2(1.950903220e-01f, -9.807852804e-01f);
    case 8: return make_float2(0.000000000e+00f, -1.000000000e+00f);
    case 9: return make_float2(-1.950903220e-01f, -9.807852804e-01f);
    case 10: return make_float2(-3.826834324e-01f, -9.238795325e-01f);
    case 11: return make_float2(-5.555702330e-01f, -8.314696123e-01f);
    case 12: return make_float2(-7.071067812e-01f, -7.071067812e-01f);
    case 13: return make_float2(-8.314696123e-01f, -5.555702330e-01f);
    case 14: return make_float2(-9.238795325e-01f, -3.826834324e-01f);
    case 15: return make_float2(-9.807852804e-01f, -1.950903220e-01f);
    case 16: return make_float2(-1.000000000e+00f, 0.000000000e+00f);
    case 17: return make_float2(-9.807852804e-01f, 1.950903220e-01f);
    case 18: return make_float2(-9.238795325e-01f, 3.826834324e-01f);
    case 19: return make_float2(-8.314696123e-01f, 5.555702330e-01f);
    case 20: return make_float2(-7.071067812e-01f, 7.071067812e-01f);
    case 21: return make_float2(-5.555702330e-01f, 8.314696123e-01f);
    case 22: return make_float2(-3.826834324e-01f, 9.238795325e-01f);
    case 23: return make_float2(-1.950903220e-01f, 9.807852804e-01f);
    case 24: return make_float2(0.000000000e+00f, 1.000000000e+00f);
    case 25: return make_float2(1.950903220e-01f, 9.807852804e-01f);
    case 26: return make_float2(3.826834324e-01f, 9.238795325e-01f);
    case 27: return make_float2(5.555702330e-01f, 8.314696123e-01f);
    case 28: return make_float2(7.071067812e-01f, 7.071067812e-01f);
    case 29: return make_float2(8.314696123e-01f, 5.555702330e-01f);
    case 30: return make_float2(9.238795325e-01f, 3.826834324e-01f);
    case 31: return make_float2(9.807852804e-01f, 1.950903220e-01f);
    default: return make_float2(1.f, 0.f);
  }
}
__device__ __forceinline__ float2 tw24(int k) {
  switch (k) {
    case 0: return make_float2(1.000000000e+00f, 0.000000000e+00f);
    case 1: return make_float2(9.659258263e-01f, -2.588190451e-01f);
    case 2: return make_float2(8.660254038e-01f, -5.000000000e-01f);
    case 3: return make_float2(7.071067812e-01f, -7.071067812e-01f);
    case 4: return make_float2(5.000000000e-01f, -8.660254038e-01f);
    case 5: return make_float2(2.588190451e-01f, -9.659258263e-01f);
    case 6: return make_float2(0.000000000e+00f, -1.000000000e+00f);
    case 7: return make_float2(-2.588190451e-01f, -9.659258263e-01f);
    case 8: return make_float2(-5.000000000e-01f, -8.660254038e-01f);
    case 9: return make_float2(-7.071067812e-01f, -7.071067812e-01f);
    case 10: return make_float2(-8.660254038e-01f, -5.000000000e-01f);
    case 11: return make_float2(-9.659258263e-01f, -2.588190451e-01f);
    case 12: return make_float2(-1.000000000e+00f, 0.000000000e+00f);
    case 13: return make_float2(-9.659258263e-01f, 2.588190451e-01f);
    case 14: return make_float2(-8.660254038e-01f, 5.000000000e-01f);
    case 15: return make_float2(-7.071067812e-01f, 7.071067812e-01f);
    case 16: return make_float2(-5.000000000e-01f, 8.660254038e-01f);
    case 17: return make_float2(-2.588190451e-01f, 9.659258263e-01f);
    case 18: return make_float2(0.000000000e+00f, 1.000000000e+00f);
    case 19: return make_float2(2.588190451e-01f, 9.659258263e-01f);
    case 20: return make_float2(5.000000000e-01f, 8.660254038e-01f);
    case 21: return make_float2(7.071067812e-01f, 7.071067812e-01f);
    case 22: return make_float2(8.660254038e-01f, 5.000000000e-01f);
    case 23: return make_float2(9.659258263e-01f, 2.588190451e-01f);
    default: return make_float2(1.f, 0.f);
  }
}

__host__ __device__ constexpr int bitrev_c(int i, int bits) {
  int r = 0;
  for (int b = 0; b < bits; ++b) r |= ((i >> b) & 1) << (bits - 1 - b);
  return r;
}
__host__ __device__ constexpr int ilog2_c(int n) { return n <= 1 ? 0 : 1 + ilog2_c(n / 2); }

// w_N^j (forward sign) for N dividing 32 or 24; conjugated for SIGN > 0
template <int N, int SIGN>
__device__ __forceinline__ float2 twr(int j) {
  float2 w;
  if (32 % N == 0) w = tw32(j * (32 / N));
  else w = tw24(j * (24 / N));
  if (SIGN > 0) w.y = -w.y;
  return w;
}

// in-register radix-2 DIT DFT, N a power of two
template <int N, int SIGN>
__device__ __forceinline__ void dft_pow2(float2 (&a)[N]) {
  constexpr int B = ilog2_c(N);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int j = bitrev_c(i, B);
    if (j > i) {
      const float2 t = a[i];
      a[i] = a[j];
      a[j] = t;
    }
  }
#pragma unroll
  for (int half = 1; half < N; half *= 2) {
#pragma unroll
    for (int k = 0; k < N; k += 2 * half) {
#pragma unroll
      for (int j = 0; j < half; ++j) {
        float2 t = a[k + j + half];
        if (j != 0) t = cmul(twr<N, SIGN>(j * (N / (2 * half))), t);
        a[k + j + half] = csub(a[k + j], t);
        a[k + j] = cadd(a[k + j], t);
      }
    }
  }
}

// N = 3 M: three interleaved DFTs of length M and a radix-3 combination
template <int M, int SIGN>
__device__ __forceinline__ void dft_3m(float2 (&a)[3 * M]) {
  constexpr int N = 3 * M;
  float2 b0[M], b1[M], b2[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    b0[m] = a[3 * m];
    b1[m] = a[3 * m + 1];
    b2[m] = a[3 * m + 2];
  }
  dft_pow2<M, SIGN>(b0);
  dft_pow2<M, SIGN>(b1);
  dft_pow2<M, SIGN>(b2);
  const float s3 = 0.86602540378443864676f * (float)SIGN;
#pragma unroll
  for (int k = 0; k < M; ++k) {
    float2 t1 = b1[k], t2 = b2[k];
    if (k != 0) {
      t1 = cmul(twr<N, SIGN>(k), t1);
      t2 = cmul(twr<N, SIGN>(2 * k), t2);
    }
    const float2 s = cadd(t1, t2), d = csub(t1, t2);
    float2 m;
    m.x = b0[k].x - 0.5f * s.x;
    m.y = b0[k].y - 0.5f * s.y;
    float2 id;  // i * SIGN * sqrt(3)/2 * d
    id.x = -s3 * d.y;
    id.y = s3 * d.x;
    a[k] = cadd(b0[k], s);
    a[k + M] = cadd(m, id);
    a[k + 2 * M] = csub(m, id);
  }
}

template <int N, int SIGN>
__device__ __forceinline__ void dft_reg(float2 (&a)[N]) {
  if constexpr (N == 12) dft_3m<4, SIGN>(a);
  else if constexpr (N == 24) dft_3m<8, SIGN>(a);
  else dft_pow2<N, SIGN>(a);
}

}  // namespace ilm
