// FP32 LGF convolution of one field (the operators and solves of a cache): the
// three passes of ilm_fft.cu for padded sizes from 2048 to 8192, with no job
// table to upload and three or four register stages per transform.
//
// A transform of L points runs on L / E threads, each with E = 16 (L = 2^a) or
// 24 (3 * 2^a) values in registers: a stage is E / R DFTs of R points (R = 4 to
// 24), a twiddle table multiplication and one exchange through shared memory
// (Stockham order, one buffer, padded by one value in 16).
//   * rows: the input values are loaded straight into the first stage's
//     registers; the last stage goes through shared memory once more for the
//     split of the real transform.
//   * columns: CW neighbouring spectral columns per CTA (whole 32-byte
//     sectors).  The forward transform's last stage leaves X[j + r L / R] with
//     the thread that needs exactly these for the first stage (of the same R)
//     of the inverse, so the spectrum is multiplied in registers and the pair
//     of transforms takes four exchanges; rows at or beyond n2 are neither
//     loaded nor stored.
// The batched passes hold a transform in two steps of up to 32 points per
// thread, which ends at 1024 points (beyond, radix-4 stages between two shared
// buffers).  Measured, us per field: 1023^2 179 -> 38, 2047^2 495 -> 152; the data
// stay in L2, the exchanges and FP32 issue bound the passes.
#include <algorithm>

#include "ilm_fftcore.cuh"

namespace ilm {
namespace {

// radices of the stages (0: none)
struct Stages {
  int e, r[4];
};
constexpr Stages stages_of(int L) {
  switch (L) {
    case 1024: return {16, {16, 8, 8, 0}};
    case 1536: return {24, {8, 8, 24, 0}};
    case 2048: return {16, {16, 16, 8, 0}};
    case 3072: return {24, {8, 8, 4, 12}};
    case 4096: return {16, {16, 16, 16, 0}};
    case 6144: return {24, {8, 8, 8, 12}};
  }
  return {0, {0, 0, 0, 0}};
}
constexpr int num_stages(int L) {
  return stages_of(L).r[3] == 0 ? 3 : 4;
}
// radix of stage s of the forward (dir = 0) or inverse (1: reversed) transform
constexpr int radix_of(int L, int s, int dir) { return stages_of(L).r[dir ? num_stages(L) - 1 - s : s]; }
constexpr int span_of(int L, int s, int dir) {  // Ns: product of the radices before
  int n = 1;
  for (int q = 0; q < s; ++q) n *= radix_of(L, q, dir);
  return n;
}
__host__ __device__ constexpr int fpos(int i) { return i + (i >> 4); }
constexpr int transform_floats2(int L) { return fpos(L - 1) + 1; }

// stage S on the registers a (a[b R + r]: element j + r L / R of DFT j = t + b L / E)
template <int L, int S, int DIR>
__device__ __forceinline__ void stage_dft(float2 (&a)[stages_of(L).e], int t, const float2* __restrict__ tw, int tws) {
  constexpr int E = stages_of(L).e, R = radix_of(L, S, DIR), Ns = span_of(L, S, DIR), T = L / E;
#pragma unroll
  for (int b = 0; b < E / R; ++b) {
    const int j = t + b * T;
    float2 x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = a[b * R + r];
    if (Ns > 1) {
      const int k = (j % Ns) * (L / (Ns * R)) * tws;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        float2 w = __ldg(tw + r * k);
        if (DIR) w.y = -w.y;
        x[r] = cmul(w, x[r]);
      }
    }
    dft_reg<R, DIR ? 1 : -1>(x);
#pragma unroll
    for (int r = 0; r < R; ++r) a[b * R + r] = x[r];
  }
}
// registers of stage S (after its DFTs) -> shared memory in Stockham order
template <int L, int S, int DIR>
__device__ __forceinline__ void stage_put(const float2 (&a)[stages_of(L).e], int t, float2* s) {
  constexpr int E = stages_of(L).e, R = radix_of(L, S, DIR), Ns = span_of(L, S, DIR), T = L / E;
#pragma unroll
  for (int b = 0; b < E / R; ++b) {
    const int j = t + b * T, base = (j / Ns) * (Ns * R) + j % Ns;
#pragma unroll
    for (int r = 0; r < R; ++r) s[fpos(base + r * Ns)] = a[b * R + r];
  }
}
template <int L, int S, int DIR>
__device__ __forceinline__ void stage_get(float2 (&a)[stages_of(L).e], int t, const float2* s) {
  constexpr int E = stages_of(L).e, R = radix_of(L, S, DIR), T = L / E;
#pragma unroll
  for (int b = 0; b < E / R; ++b)
#pragma unroll
    for (int r = 0; r < R; ++r) a[b * R + r] = s[fpos(t + b * T + r * (L / R))];
}
// stages S .. last, the first one's input in registers; on return the last
// stage's DFTs are in registers (element j + r L / R, natural order)
template <int L, int S, int DIR>
__device__ __forceinline__ void stages_from(float2 (&a)[stages_of(L).e], int t, float2* s,
                                            const float2* __restrict__ tw, int tws) {
  stage_dft<L, S, DIR>(a, t, tw, tws);
  if constexpr (S + 1 < num_stages(L)) {
    if (S > 0) __syncthreads();  // the last exchange has been read
    stage_put<L, S, DIR>(a, t, s);
    __syncthreads();
    stage_get<L, S + 1, DIR>(a, t, s);
    stages_from<L, S + 1, DIR>(a, t, s, tw, tws);
  }
}

struct FieldJob {
  const float* in;
  float* out;
  float2* work;         // n2 x (P1 / 2 + 1)
  const float* spec;    // (P1 / 2 + 1) x (P2 / 2 + 1)
  const float2* tw1;    // exp(-2 pi i m / P1)
  const float2* tw2;    // exp(-2 pi i m / P2)
  int n1, n2;
  float scale;
};

// rows: real transforms of length 2 H, a CTA of H / E threads each
template <int H>
__global__ void __launch_bounds__(H / stages_of(H).e) k_rows_field(const FieldJob J) {
  constexpr int E = stages_of(H).e, T = H / E, ns = num_stages(H);
  constexpr int R0 = radix_of(H, 0, 0), RL = radix_of(H, ns - 1, 0);
  extern __shared__ __align__(16) float2 sm_field[];
  const int t = threadIdx.x, row = blockIdx.x;
  float2* s = sm_field;
  const float* __restrict__ x = J.in + (size_t)row * J.n1;
  float2 a[E];
#pragma unroll
  for (int b = 0; b < E / R0; ++b)
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      const int m = 2 * (t + b * T + r * (H / R0));
      a[b * R0 + r] = make_float2(m < J.n1 ? __ldg(x + m) : 0.f, m + 1 < J.n1 ? __ldg(x + m + 1) : 0.f);
    }
  stages_from<H, 0, 0>(a, t, s, J.tw1, 2);
  __syncthreads();
#pragma unroll
  for (int b = 0; b < E / RL; ++b)
#pragma unroll
    for (int r = 0; r < RL; ++r) s[fpos(t + b * T + r * (H / RL))] = a[b * RL + r];
  __syncthreads();
  float2* __restrict__ W = J.work + (size_t)row * (H + 1);
  for (int k = t; k <= H; k += T) {
    const float2 zk = s[fpos(k == H ? 0 : k)];
    float2 zc = s[fpos(k == 0 ? 0 : H - k)];
    zc.y = -zc.y;
    const float2 e = __ldg(J.tw1 + k);
    const float2 p = cadd(zk, zc), d = csub(zk, zc);
    const float2 ed = cmul(e, d);
    W[k] = make_float2(0.5f * (p.x + ed.y), 0.5f * (p.y - ed.x));
  }
}

template <int H>
__global__ void __launch_bounds__(H / stages_of(H).e) k_irows_field(const FieldJob J) {
  constexpr int E = stages_of(H).e, T = H / E, ns = num_stages(H);
  constexpr int R0 = radix_of(H, 0, 1), RL = radix_of(H, ns - 1, 1);
  extern __shared__ __align__(16) float2 sm_field[];
  const int t = threadIdx.x, row = blockIdx.x;
  const float2* __restrict__ W = J.work + (size_t)row * (H + 1);
  float2 a[E];
#pragma unroll
  for (int b = 0; b < E / R0; ++b)
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      const int k = t + b * T + r * (H / R0);
      const float2 xk = W[k];
      float2 xc = W[H - k];
      xc.y = -xc.y;
      float2 e = __ldg(J.tw1 + k);
      e.y = -e.y;
      const float2 p = cadd(xk, xc), d = csub(xk, xc);
      const float2 ed = cmul(e, d);
      a[b * R0 + r] = make_float2(0.5f * (p.x - ed.y), 0.5f * (p.y + ed.x));
    }
  stages_from<H, 0, 1>(a, t, sm_field, J.tw1, 2);
  float* __restrict__ o = J.out + (size_t)row * J.n1;
#pragma unroll
  for (int b = 0; b < E / RL; ++b)
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      const int m = 2 * (t + b * T + r * (H / RL));
      if (m < J.n1) o[m] = a[b * RL + r].x * J.scale;
      if (m + 1 < J.n1) o[m + 1] = a[b * RL + r].y * J.scale;
    }
}

// spectral columns per CTA: 4 (a 32-byte sector of every row) where that is at
// most 512 threads, so that a thread's values stay in registers, else 2
constexpr int field_cw(int L) { return 4 * (L / stages_of(L).e) <= 512 ? 4 : 2; }
// stride of a column's buffer: 4 (mod 16) for four columns side by side in a
// half-warp, 8 for two (with the pad of fpos the 16 lanes hit 16 bank pairs)
constexpr int field_cs(int L) {
  int c = transform_floats2(L);
  while (c % 16 != (field_cw(L) == 4 ? 4 : 8)) ++c;
  return c;
}

template <int L>
__global__ void __launch_bounds__(field_cw(L) * (L / stages_of(L).e)) k_cols_field(const FieldJob J, int ncols) {
  constexpr int E = stages_of(L).e, T = L / E, ns = num_stages(L), CW = field_cw(L), CS = field_cs(L);
  constexpr int R0 = radix_of(L, 0, 0), RL = radix_of(L, ns - 1, 0);  // RL: also the inverse's first radix
  extern __shared__ __align__(16) float2 sm_field[];
  const int c = threadIdx.x % CW, t = threadIdx.x / CW, col = blockIdx.x * CW + c;
  const bool act = col < ncols;
  float2* s = sm_field + c * CS;
  float2* __restrict__ W = J.work + (act ? col : 0);
  float2 a[E];
#pragma unroll
  for (int b = 0; b < E / R0; ++b)
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      const int row = t + b * T + r * (L / R0);
      a[b * R0 + r] = act && row < J.n2 ? W[(size_t)row * ncols] : make_float2(0.f, 0.f);
    }
  stages_from<L, 0, 0>(a, t, s, J.tw2, 1);
  const float* __restrict__ spec = J.spec + (size_t)(act ? col : 0) * (L / 2 + 1);
#pragma unroll
  for (int b = 0; b < E / RL; ++b)
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      const int k = t + b * T + r * (L / RL);
      const float sv = __ldg(spec + (k <= L - k ? k : L - k));
      a[b * RL + r].x *= sv;
      a[b * RL + r].y *= sv;
    }
  __syncthreads();  // the forward transform's last exchange has been read
  stages_from<L, 0, 1>(a, t, s, J.tw2, 1);
  if (!act) return;
  // the inverse ends with radix R0
#pragma unroll
  for (int b = 0; b < E / R0; ++b)
#pragma unroll
    for (int r = 0; r < R0; ++r) {
      const int row = t + b * T + r * (L / R0);
      if (row < J.n2) W[(size_t)row * ncols] = a[b * R0 + r];
    }
}

template <typename K>
int run(K kernel, int grid, int threads, size_t smem, const FieldJob& J, cudaStream_t st) {
  ILM_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<grid, threads, smem, st>>>(J);
  ILM_CHECK_LAUNCH();
  return ILM_OK;
}

template <int H>
int run_rows(const FieldJob& J, bool inverse, cudaStream_t st) {
  constexpr int T = H / stages_of(H).e;
  const size_t smem = transform_floats2(H) * sizeof(float2);
  return inverse ? run(k_irows_field<H>, J.n2, T, smem, J, st) : run(k_rows_field<H>, J.n2, T, smem, J, st);
}

template <int L>
int run_cols(const FieldJob& J, int ncols, cudaStream_t st) {
  constexpr int CW = field_cw(L);
  const size_t smem = (size_t)CW * field_cs(L) * sizeof(float2);
  ILM_CHECK_CUDA(cudaFuncSetAttribute(k_cols_field<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_cols_field<L><<<(ncols + CW - 1) / CW, CW * (L / stages_of(L).e), smem, st>>>(J, ncols);
  ILM_CHECK_LAUNCH();
  return ILM_OK;
}

int rows_any(int H, const FieldJob& J, bool inverse, cudaStream_t st) {
  switch (H) {
    case 1024: return run_rows<1024>(J, inverse, st);
    case 1536: return run_rows<1536>(J, inverse, st);
    case 2048: return run_rows<2048>(J, inverse, st);
    case 3072: return run_rows<3072>(J, inverse, st);
    case 4096: return run_rows<4096>(J, inverse, st);
  }
  return ILM_ERR_UNSUPPORTED;
}

int cols_any(int L, const FieldJob& J, int ncols, cudaStream_t st) {
  switch (L) {
    case 2048: return run_cols<2048>(J, ncols, st);
    case 3072: return run_cols<3072>(J, ncols, st);
    case 4096: return run_cols<4096>(J, ncols, st);
    case 6144: return run_cols<6144>(J, ncols, st);
  }
  return ILM_ERR_UNSUPPORTED;
}

}  // namespace

// P1 / 2 and P2 are 2^a or 3 * 2^a (good_fft_size).  Below 2048 points the passes
// of ilm_fft.cu stay although these would be faster (405^2 37 and 19 us, 600^2 92
// and 31): where a result cancels (the surface values of a smooth double layer on
// one nearly circular body are 1/200 of the field), another order of the FP32
// roundings moves it by up to 2e-4 there, by some 1e-5 from 2048 points on; the
// errors against 64 bits are the same.
bool field_conv_supported(int P1, int P2) {
  const int H = P1 / 2;
  return H >= 1024 && H <= 4096 && P2 >= 2048 && P2 <= 6144;
}

int field_conv_apply(ConvPlan* p, const float* in, float* out, double scale, cudaStream_t st) {
  const FieldJob J{in,
                  out,
                  p->work.as<float2>(),
                  static_cast<const float*>(p->spec),
                  static_cast<const float2*>(p->tw1),
                  static_cast<const float2*>(p->tw2),
                  p->n1,
                  p->n2,
                  (float)scale};
  const int H = p->P1 / 2;
  ILM_TRY(rows_any(H, J, false, st));
  ILM_TRY(cols_any(p->P2, J, H + 1, st));
  return rows_any(H, J, true, st);
}

}  // namespace ilm
