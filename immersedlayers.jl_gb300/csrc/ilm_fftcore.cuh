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

}  // namespace ilm
