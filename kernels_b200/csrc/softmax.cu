// Row softmax  y = exp(x - max) / sum  over the last axis of a [rows, cols] matrix.
//
// HBM-bound: every element is read once and written once (2 * rows * cols * elsize bytes),
// so the kernel keeps a whole row in registers between the reduction and the store and
// moves data in 16-byte vectors with streaming cache hints.
//   * cols <= 32 * 16-byte vectors * 8 : one warp per row, several rows per CTA;
//   * cols <= 512 threads * 8 vectors (fp32: 1024 threads): one CTA per row, block reduction through smem;
//   * rows that start off a 16-byte boundary (an odd row length): the same kernels, the row cut into the elements
//     before its first boundary, 16-byte vectors and the elements after its last one;
//   * otherwise (longer rows, or x and y rows at different offsets from a boundary): a three-pass scalar kernel.
// Reference semantics: src/softmax/kernel.py:27-91 (natural exponent, fp32 math).
#include <math.h>

#include <type_traits>

#include "common.cuh"

namespace kb {
namespace {

template <typename T>
struct Vec16 {
  static constexpr int kElems = 16 / sizeof(T);
};

template <typename T>
__device__ __forceinline__ void expand_vec(const int4& raw, float (&out)[Vec16<T>::kElems]) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < Vec16<T>::kElems; ++i) out[i] = to_f32(e[i]);
}

// The compiler must not carry what it derived from the words across this point (it would keep, and spill, the
// expanded values instead of expanding them again).
__device__ __forceinline__ void forget(int4& raw) { asm volatile("" : "+r"(raw.x), "+r"(raw.y), "+r"(raw.z), "+r"(raw.w)); }

template <typename T>
__device__ __forceinline__ void store_vec(T* p, const float (&in)[Vec16<T>::kElems]) {
  int4 raw;
  T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int i = 0; i < Vec16<T>::kElems; ++i) e[i] = from_f32<T>(in[i]);
  __stcs(reinterpret_cast<int4*>(p), raw);
}

__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// One row per GROUP threads (GROUP = 32: warp per row; GROUP = blockDim: CTA per row).
// Each thread holds NV 16-byte vectors of its row; vector v of thread t covers elements
// (v * GROUP + t) * kElems .. +kElems, so a warp's accesses are contiguous.
//
// RAGGED: rows may start anywhere (x and y at the same offset from a 16-byte boundary).  Up to kElems - 1 elements
// before the first boundary and after the last one are held one each by the first 2 kElems threads of the row.  For
// fp32 the exponent is formed as x - max before the multiplication, as in the scalar kernel.
//
// Eight vectors of 16-bit elements are 64 fp32 values: with those a CTA of 512 threads had the SM to itself and a row's
// loads overlapped nothing (bf16 [8011, 19992]: 275 us, 2.3 TB/s).  They stay packed instead and are expanded, and
// their exponentials evaluated, once for the sum and once for the store (the same value both times).  64 registers
// per thread are the cap of the CTA-per-row instances: 1024 threads' worth of rows are in flight on every SM.
template <typename T, int NV, int GROUP, int THREADS, bool RAGGED>
__global__ void __launch_bounds__(THREADS, GROUP > 32 ? 1024 / THREADS : 2) softmax_rows_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                               int64_t rows, int cols, int64_t xs, int64_t ys) {
  constexpr int E = Vec16<T>::kElems;
  constexpr int ROWS_PER_CTA = THREADS / GROUP;
  __shared__ float red[THREADS / 32];
  const int lane_in_group = threadIdx.x % GROUP;
  const int64_t row = (int64_t)blockIdx.x * ROWS_PER_CTA + threadIdx.x / GROUP;
  const bool row_ok = row < rows;
  const T* xr = x + (row_ok ? row : 0) * xs;
  T* yr = y + (row_ok ? row : 0) * ys;

  int head = 0, body = cols, edge = -1;  // elements before the first boundary, in vectors; this thread's edge element
  if (RAGGED) {
    const int off = (int)(reinterpret_cast<uintptr_t>(xr) & 15);
    head = off ? min((16 - off) / (int)sizeof(T), cols) : 0;
    body = (cols - head) / E * E;
    if (lane_in_group < head) edge = lane_in_group;
    else if (lane_in_group >= E && lane_in_group - E < cols - head - body) edge = head + body + lane_in_group - E;
    if (!row_ok) edge = -1;
  }
  constexpr bool kPacked = sizeof(T) == 2 && NV == 8 && GROUP > 32;
  constexpr uint32_t kNegInf = sizeof(T) == 4 ? 0xff800000u : (std::is_same<T, __half>::value ? 0xfc00fc00u : 0xff80ff80u);
  int4 raw[NV];
  float v[kPacked ? 1 : NV][E], ve = -INFINITY;
  float mx = -INFINITY;
  if (RAGGED) {
    if (edge >= 0) ve = to_f32(xr[edge]);
    mx = fmaxf(mx, ve);
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (i * GROUP + lane_in_group) * E;
    raw[i] = row_ok && col < body ? __ldcs(reinterpret_cast<const int4*>(xr + head + col)) : make_int4(kNegInf, kNegInf, kNegInf, kNegInf);
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float (&f)[E] = v[kPacked ? 0 : i];
    expand_vec<T>(raw[i], f);
#pragma unroll
    for (int e = 0; e < E; ++e) mx = fmaxf(mx, f[e]);
  }
  mx = warp_max(mx);
  if (GROUP > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) mx = fmaxf(mx, red[w]);
    __syncthreads();
  }
  // exp(z - max) with one rounding: 2^(z log2e - max log2e).  The rounding of max log2e is a factor that the whole row
  // shares, and cancels as long as it stays near 1: up to |max| = 2^16 it lies within 2^(2^-8) of it, from 2^31 on it alone
  // leaves fp32's range.  A larger maximum (of a row masked to the type's lowest value, an infinity) is subtracted first: in
  // fp32 from the values held, in the rare row that has one.  In bf16 all that is not the maximum then lies 256 or more
  // below it and counts as 0 in any base, so base 2 does, which is another multiplier and no branch: rows of 130-1003
  // elements, 40 MB in L2, 34.6 / 17.6 / 13.9 / 13.2 us without the check, 35.1 / 17.7 / 14.0 / 13.5 with it (with fp32's branch
  // 35.9 / 18.4 / 14.2 / 13.3).  Finite fp16 values never come to that, and the odd-length fp32 rows subtract anyway.
  constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
  const bool far = (kBf16 || (sizeof(T) == 4 && !RAGGED)) && !(fabsf(mx) <= 65536.f);
  const float mul = kBf16 && far ? 1.f : kLog2e;
  float shift = kBf16 && far ? mx : mx * kLog2e;
  if (!kBf16 && __builtin_expect(far, 0)) {
#pragma unroll
    for (int i = 0; i < (kPacked ? 1 : NV); ++i)
#pragma unroll
      for (int e = 0; e < E; ++e) v[i][e] -= mx;
    shift = 0.f;
  }
  auto exp_of = [&](float z) { return RAGGED && sizeof(T) == 4 ? expf(z - mx) : exp2f(fmaf(z, mul, -shift)); };
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float (&f)[E] = v[kPacked ? 0 : i];
    if (kPacked) {
      forget(raw[i]);
      expand_vec<T>(raw[i], f);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      f[e] = exp_of(f[e]);
      sum += f[e];
    }
  }
  if (RAGGED && edge >= 0) {
    ve = exp_of(ve);
    sum += ve;
  }
  sum = warp_sum(sum);
  if (GROUP > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    sum = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) sum += red[w];
  }
  const float inv = 1.f / sum;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (i * GROUP + lane_in_group) * E;
    if (row_ok && col < body) {
      float (&f)[E] = v[kPacked ? 0 : i];
      if (kPacked) {
        forget(raw[i]);
        expand_vec<T>(raw[i], f);
      }
#pragma unroll
      for (int e = 0; e < E; ++e) f[e] = (kPacked ? exp_of(f[e]) : f[e]) * inv;
      store_vec<T>(yr + head + col, f);
    }
  }
  if (RAGGED && edge >= 0) yr[edge] = from_f32<T>(ve * inv);
}

// Any shape / alignment: one CTA per row, three passes over the row (max, sum, write).
template <typename T>
__global__ void __launch_bounds__(256) softmax_rows_scalar_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                                  int64_t cols, int64_t xs, int64_t ys) {
  __shared__ float red[8];
  const T* xr = x + (int64_t)blockIdx.x * xs;
  T* yr = y + (int64_t)blockIdx.x * ys;
  float mx = -INFINITY;
  for (int64_t i = threadIdx.x; i < cols; i += 256) mx = fmaxf(mx, to_f32(xr[i]));
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = red[0];
  for (int w = 1; w < 8; ++w) mx = fmaxf(mx, red[w]);
  __syncthreads();
  float sum = 0.f;
  for (int64_t i = threadIdx.x; i < cols; i += 256) sum += expf(to_f32(xr[i]) - mx);
  sum = warp_sum(sum);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  sum = 0.f;
  for (int w = 0; w < 8; ++w) sum += red[w];
  const float inv = 1.f / sum;
  for (int64_t i = threadIdx.x; i < cols; i += 256) yr[i] = from_f32<T>(expf(to_f32(xr[i]) - mx) * inv);
}

template <typename T, int NV, int GROUP, int THREADS, bool RAGGED>
int launch_vec(const kb_softmax_params& p, cudaStream_t s) {
  constexpr int rows_per_cta = THREADS / GROUP;
  const int64_t ctas = (p.rows + rows_per_cta - 1) / rows_per_cta;
  softmax_rows_kernel<T, NV, GROUP, THREADS, RAGGED><<<(unsigned)ctas, THREADS, 0, s>>>(
      static_cast<const T*>(p.x), static_cast<T*>(p.y), p.rows, (int)p.cols, p.x_row_stride, p.y_row_stride);
  KB_LAUNCH_CHECK("softmax_rows_kernel");
  return KB_OK;
}

// KB_ERR_UNSUPPORTED: no instance holds so long a row
template <typename T, bool RAGGED>
int launch_by_length(const kb_softmax_params& p, cudaStream_t s) {
  const int64_t vecs = p.cols / Vec16<T>::kElems;
  if (vecs <= 32 * 1) return launch_vec<T, 1, 32, 256, RAGGED>(p, s);
  if (vecs <= 32 * 2) return launch_vec<T, 2, 32, 256, RAGGED>(p, s);
  if (vecs <= 32 * 4) return launch_vec<T, 4, 32, 256, RAGGED>(p, s);
  if (vecs <= 32 * 8) return launch_vec<T, 8, 32, 256, RAGGED>(p, s);
  if (vecs <= 256 * 2) return launch_vec<T, 2, 256, 256, RAGGED>(p, s);
  if (vecs <= 256 * 4) return launch_vec<T, 4, 256, 256, RAGGED>(p, s);
  if (vecs <= 256 * 8) return launch_vec<T, 8, 256, 256, RAGGED>(p, s);
  if (vecs <= 512 * 8) return launch_vec<T, 8, 512, 512, RAGGED>(p, s);
  // 1024 threads leave 64 registers each: enough for eight vectors of fp32, not of 16-bit elements
  if constexpr (RAGGED && sizeof(T) == 4) {
    if (vecs <= 1024 * 8) return launch_vec<T, 8, 1024, 1024, RAGGED>(p, s);
  }
  return KB_ERR_UNSUPPORTED;
}

template <typename T>
int softmax_typed(const kb_softmax_params& p, cudaStream_t s) {
  constexpr int E = Vec16<T>::kElems;
  const bool aligned = (reinterpret_cast<uintptr_t>(p.x) % 16 == 0) && (reinterpret_cast<uintptr_t>(p.y) % 16 == 0) &&
                       (p.x_row_stride % E == 0) && (p.y_row_stride % E == 0) && (p.cols % E == 0);
  // every x row lies as far from a 16-byte boundary as its y row (elements on their natural boundaries)
  const bool in_step = (reinterpret_cast<uintptr_t>(p.x) - reinterpret_cast<uintptr_t>(p.y)) % 16 == 0 &&
                       reinterpret_cast<uintptr_t>(p.x) % sizeof(T) == 0 && (p.x_row_stride - p.y_row_stride) % E == 0;
  if (p.rows < (int64_t)1 << 31 && (aligned || in_step)) {
    // The aligned instances end at 512 threads; a longer aligned row is a ragged one without edges.
    const int rc = aligned && p.cols / E <= 512 * 8 ? launch_by_length<T, false>(p, s) : launch_by_length<T, true>(p, s);
    if (rc != KB_ERR_UNSUPPORTED) return rc;
  }
  if (p.rows >= (int64_t)1 << 31) return KB_ERR_TOO_LARGE;
  softmax_rows_scalar_kernel<T><<<(unsigned)p.rows, 256, 0, s>>>(static_cast<const T*>(p.x), static_cast<T*>(p.y),
                                                                p.cols, p.x_row_stride, p.y_row_stride);
  KB_LAUNCH_CHECK("softmax_rows_scalar_kernel");
  return KB_OK;
}

}  // namespace

int softmax_rows(const kb_softmax_params& p, cudaStream_t s) {
  if (p.rows == 0 || p.cols == 0) return KB_OK;
  switch (p.dtype) {
    case KB_F32: return softmax_typed<float>(p, s);
    case KB_F16: return softmax_typed<__half>(p, s);
    case KB_BF16: return softmax_typed<__nv_bfloat16>(p, s);
    default: return KB_ERR_UNSUPPORTED;
  }
}

}  // namespace kb
