// Quantisation of a [B, H, T, 128] tensor to e4m3 with one fp32 scale per tile of 128 rows: what the 8-bit
// forward takes.  scale = max(|x| of the tile) * (1 / 448), at least 1e-12; x8 = e4m3(x / scale).
//
// HBM-bound: every element is read once and written once as a byte (16-bit input: 3 bytes per element).  One CTA
// owns a tile (32 KB of 16-bit, 64 KB of fp32 input) and keeps it in registers between the maximum and the
// conversion, eight 16-byte vectors per thread, all loads in flight at once; several CTAs per SM overlap one
// tile's reduction with another's loads.
//
// The maximum is taken over the bit patterns without the sign: for non-negative floats they order like the
// values, and a NaN orders above every number, so it reaches the scale as it does in a floating-point maximum
// that propagates NaN.
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace kb {
namespace {

constexpr int kRows = 128, kD = 128, kVecs = 8;

template <typename T>
struct QuantTraits {
  static constexpr int kElems = 16 / sizeof(T);                              // per 16-byte vector
  static constexpr int kThreads = kRows * kD / (kElems * kVecs);             // 256 (16-bit), 512 (fp32)
};

struct QuantArgs {
  const void* x;
  uint8_t* x8;
  float* scale;
  int64_t sb, sh, st;
  int32_t H, T, n;
  KbFastDiv fd_n, fd_H;
};

__device__ __forceinline__ uint32_t abs_bits_max(uint32_t m, float, uint32_t w) { return max(m, w & 0x7fffffffu); }
template <typename T>
__device__ __forceinline__ uint32_t abs_bits_max(uint32_t m, T, uint32_t w) { return __vmaxu2(m, w & 0x7fff7fffu); }

// x / scale rounded to nearest, with r = 1 / scale rounded to nearest: one Newton correction of x r by its exact
// remainder (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990: correctly
// rounded where nothing underflows).  Here scale >= 1e-12 and quotients below 2^-11 become 0 whatever their last bit,
// so the remainders that matter stay far above the smallest normal number; scale <= 1e37 keeps r normal.
__device__ __forceinline__ float div_by(float x, float scale, float r) {
  const float q = __fmul_rn(x, r);
  const float d = __fmaf_rn(__fmaf_rn(-q, scale, x), r, q);
  return __uint_as_float(__float_as_uint(d) | (__float_as_uint(x) & 0x80000000u));  // -0 keeps its sign
}

template <typename T>
__global__ void __launch_bounds__(QuantTraits<T>::kThreads) quantize_fp8_tiles_kernel(const QuantArgs a) {
  constexpr int E = QuantTraits<T>::kElems, kThreads = QuantTraits<T>::kThreads, kVecsPerRow = kD / E;
  __shared__ uint32_t red[kThreads / 32];
  const int tile = blockIdx.x;
  const int bh = kb_fastdiv(tile, a.fd_n), t0 = (tile - bh * a.n) * kRows;
  const int b = kb_fastdiv(bh, a.fd_H), h = bh - b * a.H;
  const T* x = static_cast<const T*>(a.x) + b * a.sb + h * a.sh;
  const int rows = kb_min_i32(kRows, a.T - t0);

  uint4 v[kVecs];
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int idx = i * kThreads + threadIdx.x, r = idx / kVecsPerRow, d = (idx - r * kVecsPerRow) * E;
    v[i] = r < rows ? __ldcs(reinterpret_cast<const uint4*>(x + (int64_t)(t0 + r) * a.st + d)) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int i = 0; i < kVecs; ++i)
    m = abs_bits_max(abs_bits_max(abs_bits_max(abs_bits_max(m, T(), v[i].x), T(), v[i].y), T(), v[i].z), T(), v[i].w);
  // as the bits of a float from here on
  if (sizeof(T) == 2) {
    const uint16_t hw = (uint16_t)max(m & 0xffffu, m >> 16);
    m = __float_as_uint(to_f32(*reinterpret_cast<const T*>(&hw)));
  }
  m = __reduce_max_sync(0xffffffffu, m & 0x7fffffffu);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) m = max(m, red[w]);
  const float amax = __uint_as_float(m);
  float scale = __fmul_rn(amax, 1.f / 448.f);
  if (scale < 1e-12f) scale = 1e-12f;  // (a NaN stays)
  if (threadIdx.x == 0) a.scale[tile] = scale;

  const float r = 1.f / scale;
  const bool finite = scale <= 1e37f;  // of a tile of finite numbers: at most 2^128 / 448
  uint8_t* out = a.x8 + ((int64_t)bh * a.T + t0) * kD;
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int idx = i * kThreads + threadIdx.x, row = idx / kVecsPerRow, d = (idx - row * kVecsPerRow) * E;
    if (row >= rows) continue;
    const T* e = reinterpret_cast<const T*>(&v[i]);
    uint32_t w[E / 4];
    if (finite) {
#pragma unroll
      for (int j = 0; j < E / 4; ++j)
        w[j] = sm100::pack_e4m3x4(div_by(to_f32(e[4 * j]), scale, r), div_by(to_f32(e[4 * j + 1]), scale, r),
                                  div_by(to_f32(e[4 * j + 2]), scale, r), div_by(to_f32(e[4 * j + 3]), scale, r));
    } else {  // an infinity or a NaN in the tile
#pragma unroll
      for (int j = 0; j < E / 4; ++j)
        w[j] = sm100::pack_e4m3x4(to_f32(e[4 * j]) / scale, to_f32(e[4 * j + 1]) / scale, to_f32(e[4 * j + 2]) / scale, to_f32(e[4 * j + 3]) / scale);
    }
    if (E == 8) *reinterpret_cast<uint2*>(out + row * kD + d) = make_uint2(w[0], w[E / 4 - 1]);
    else *reinterpret_cast<uint32_t*>(out + row * kD + d) = w[0];
  }
}

template <typename T>
int launch(const kb_quantize_fp8_params& p, cudaStream_t s) {
  const int64_t st[3] = {p.x.stride[0], p.x.stride[1], p.x.stride[2]};
  constexpr int E = QuantTraits<T>::kElems;
  if (p.x.stride[3] != 1 || reinterpret_cast<uintptr_t>(p.x.data) % 16 || reinterpret_cast<uintptr_t>(p.x8) % 16 || st[0] % E || st[1] % E ||
      st[2] % E)
    return KB_ERR_UNSUPPORTED;
  QuantArgs a;
  a.x = p.x.data;
  a.x8 = static_cast<uint8_t*>(p.x8);
  a.scale = p.scale;
  a.sb = st[0], a.sh = st[1], a.st = st[2];
  a.H = p.H, a.T = p.T, a.n = kb_cdiv_i32(p.T, kRows);
  a.fd_n = kb_fastdiv_make(a.n);
  a.fd_H = kb_fastdiv_make(p.H);
  const int64_t tiles = (int64_t)p.B * p.H * a.n;
  if (tiles > (int64_t)1 << 30) return KB_ERR_TOO_LARGE;
  quantize_fp8_tiles_kernel<T><<<(unsigned)tiles, QuantTraits<T>::kThreads, 0, s>>>(a);
  KB_LAUNCH_CHECK("quantize_fp8_tiles_kernel");
  return KB_OK;
}

}  // namespace

int quantize_fp8(const kb_quantize_fp8_params& p, cudaStream_t s) {
  if (p.D != kD) return KB_ERR_UNSUPPORTED;
  switch (p.dtype) {
    case KB_F32: return launch<float>(p, s);
    case KB_F16: return launch<__half>(p, s);
    case KB_BF16: return launch<__nv_bfloat16>(p, s);
    default: return KB_ERR_UNSUPPORTED;
  }
}

}  // namespace kb
