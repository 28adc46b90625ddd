// Generic CUDA-core path of streaming attention (forward, dQ pass, dK/dV pass).
//
// Covers every case the reference accepts: fp32/fp16/bf16, head_dim 16..256, arbitrary
// element strides on every input, any context size (non powers of two, larger than T) and
// any look-back.  All arithmetic is IEEE fp32 (the reference's precision="ieee" for fp32
// inputs forbids TF32).  The fp16/bf16 hot shapes are served by the tcgen05 kernels; this
// file is what runs everywhere else.
//
// Work split: one CTA owns one tile of BM query rows (forward, dQ) or BN key rows (dK/dV) of
// one (batch, head) and walks only the live tiles of the streaming schedule (schedule.h).
// Bound: the fp32 FMA pipe, then shared-memory bandwidth.  Threads form a TY x 16 grid; thread
// (ty, tx) owns the stationary rows ty + TY*i and the streamed columns tx + 16*j of a score block.
//   * Scores (A B^T): both operands are read along the head dimension, four elements per load, and
//     the products are packed fp32 pairs (fma.rn.f32x2: even and odd elements of the head dimension
//     accumulate side by side), so an 8 x 4 block costs 12 16-byte loads and 64 instructions per four
//     head-dim elements.
//   * The second matmul (P V, dS K, P dO, dS Q): the block goes through shared memory transposed,
//     [streamed column][stationary row], a thread's rows next to each other, so that a row PAIR is one
//     operand of the packed product and only the other operand has to be duplicated.
// 8 x 4 blocks of 128 threads up to head dim 64 (three / two CTAs per SM); larger head dims leave room for one
// CTA per SM and take 256 threads with half the rows each.  Measured on B200 (fp32, B=16 H=4 T=2000 D=64 c=32 back=4,
// lengths 1000-2000): forward 238 -> 145 us, dQ 336 -> 202 us, dK/dV 618 -> 260 us against 4 x 4 blocks of 256
// threads with one product per instruction, scalar loads and a division per mask element; 31-35 TFLOP/s of the
// blocks' arithmetic.  Tiles come in with cp.async where the rows
// are fp32, 16-byte aligned and dense: in the forward and the dQ pass the next tile of an operand while the block still works
// on the other; the dK/dV pass asks for Q and dO and waits for them (one buffer each).
//
// Backward: the dQ pass and the dK/dV pass each evaluate the scores and dP.  fp32 calls with a dS scratch evaluate them
// once instead: delta, dK/dV (which saves its dS tiles), dQ = dS K (sa_bwd_dq_saved_generic_kernel).  Same case: 202 +
// 260 -> 11 + 264 + 65 us.
//
// Reference semantics followed: src/streaming_attention/kernel.py:205-430 (forward),
// 639-773 and 941-1023 (dQ), 777-937 and 1027-1129 (dK/dV), 453-514 (delta).
#include <math.h>

#include "common.cuh"
#include "sm100_host.h"
#include "sm100_ptx.cuh"
#include "tiles.h"

namespace kb {
namespace {

constexpr int kPad = 4;  // floats of row padding: keeps float4 alignment, spreads banks

// tile rows and thread grid by head dim (see above)
template <int D>
struct Cfg {
  static constexpr int BM = tiles::generic_tile(D), BN = BM;
  static constexpr int TY = D <= 64 ? 8 : 16;
  static constexpr int kThreads = TY * 16;
  static constexpr int LD = D + kPad;   // row stride of an operand tile, floats
  static constexpr int PLD = BM + kPad; // row stride of a transposed score block
  static constexpr int RM = BM / TY, RN = BN / 16, DV = D / 16;
  static constexpr int VEC = DV < 4 ? DV : 4, NG = DV / VEC;  // a thread's head-dim columns: g*16*VEC + tx*VEC + e
  static constexpr int kCtasFwd = D <= 64 ? 3 : 1, kCtasBwd = D <= 64 ? 2 : 1;
};

template <typename T>
struct TensorArg {
  const T* p;
  int64_t sb, sh, st, sd;
  bool vec;  // rows are dense fp32 and 16-byte aligned: cp.async takes them
};

template <typename T>
TensorArg<T> make_arg(const kb_tensor4& t) {
  const bool vec = sizeof(T) == 4 && reinterpret_cast<uintptr_t>(t.data) % 16 == 0 && t.stride[3] == 1 && t.stride[0] % 4 == 0 &&
                   t.stride[1] % 4 == 0 && t.stride[2] % 4 == 0;
  return TensorArg<T>{static_cast<const T*>(t.data), t.stride[0], t.stride[1], t.stride[2], t.stride[3], vec};
}

template <typename T>
struct FwdArgs {
  TensorArg<T> q, k, v;
  T* o;
  float* lse;
  const int32_t* lens;
  int64_t lens_stride;
  int32_t H, T_, c, back;
  float scale_log2;
};

template <typename T>
struct BwdArgs {
  TensorArg<T> q, k, v, o, d_o;
  const float* lse;
  T* dq;
  T* dk;
  T* dv;
  float* delta;
  float* ds;  // dS scratch (single evaluation): tile (b, h, key tile, slot) of BM x BN floats
  int32_t W;  // its slots per key tile
  const int32_t* lens;
  int64_t lens_stride;
  int32_t H, T_, c, back;
  float scale_log2, sm_scale;
};

// Most query tiles a key tile meets (the schedule with len = T; a shorter sequence only clips it).
inline int32_t ds_slots(int32_t T, int32_t tile, int32_t c, int32_t back) {
  int32_t w = 1;
  for (int32_t k0 = 0; k0 < T; k0 += tile) {
    const KbTileRange r = kb_bwd_q_range(k0, tile, tile, T, c, back);
    w = kb_max_i32(w, r.end - r.begin);
  }
  return w;
}
template <int D, typename T>
__device__ __forceinline__ float* ds_tile(const BwdArgs<T>& a, int64_t bh, int kt, int slot) {
  constexpr int BM = Cfg<D>::BM;
  return a.ds + ((bh * kb_cdiv_i32(a.T_, BM) + kt) * a.W + slot) * (int64_t)(BM * BM);
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// [ROWS x D] tile of one (b, h) slice -> shared memory as fp32; rows past T read as zero.  Asynchronous (one
// cp.async group, committed here) for dense aligned fp32 rows, otherwise done when it returns.
template <int D, int ROWS, typename T>
__device__ __forceinline__ void load_tile(float* dst, const TensorArg<T>& a, int b, int h, int row0, int T_) {
  constexpr int LD = Cfg<D>::LD, kThreads = Cfg<D>::kThreads;
  const T* slice = a.p + b * a.sb + h * a.sh;
  if (sizeof(T) == 4 && a.vec) {
#pragma unroll 4
    for (int idx = threadIdx.x; idx < ROWS * (D / 4); idx += kThreads) {
      const int r = idx / (D / 4), d = (idx - r * (D / 4)) * 4, t = row0 + r;
      const bool in = t < T_;
      const T* src = slice + (in ? (int64_t)t * a.st + d : 0);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sm100::smem_u32(dst + r * LD + d)), "l"(src), "r"(in ? 16 : 0)
                   : "memory");
    }
  } else if (sizeof(T) == 4) {
    for (int idx = threadIdx.x; idx < ROWS * D; idx += kThreads) {
      const int r = idx / D, d = idx - r * D, t = row0 + r;
      dst[r * LD + d] = t < T_ ? to_f32(slice[(int64_t)t * a.st + (int64_t)d * a.sd]) : 0.f;
    }
  } else {
    // A thread stays in one column and steps over the rows.  The loads carry no condition (a row past T reads row T - 1
    // and is dropped), so that 16 of them are in flight: behind a condition 16-bit loads go one by one, which half the
    // threads per CTA had made slower.  fp16, forward + backward kernels, B=8 H=4 T=2000 c=32 back=4 / B=1 H=2 T=100: D=32
    // 313 -> 224 / 68 -> 41 us (295 / 50 with 256 threads and 4 x 4 blocks), D=16 204 -> 160 / 46 -> 32, D=256 2412 -> 1943 /
    // 142 -> 112.
    static_assert(kThreads % D == 0 && (ROWS * D) % kThreads == 0, "whole rows per step");
    constexpr int kStep = kThreads / D;
    const int d = threadIdx.x % D, r0 = threadIdx.x / D;
    const T* col = slice + (int64_t)d * a.sd;
#pragma unroll 16
    for (int i = 0; i < ROWS / kStep; ++i) {
      const int r = r0 + i * kStep, t = row0 + r;
      const float x = to_f32(col[(int64_t)kb_min_i32(t, T_ - 1) * a.st]);
      dst[r * LD + d] = t < T_ ? x : 0.f;
    }
  }
  cp_async_commit();
}

// acc[i][j] = sum_d A[ty + TY i][d] * Bm[tx + 16 j][d]
template <int D>
__device__ __forceinline__ void tile_abt(const float* A, const float* Bm, float (&acc)[Cfg<D>::RM][Cfg<D>::RN], int ty, int tx) {
  using C = Cfg<D>;
  uint64_t acc2[C::RM][C::RN];
#pragma unroll
  for (int i = 0; i < C::RM; ++i)
#pragma unroll
    for (int j = 0; j < C::RN; ++j) acc2[i][j] = 0ull;
#pragma unroll 2
  for (int d = 0; d < D; d += 4) {
    ulonglong2 a[C::RM], b[C::RN];
#pragma unroll
    for (int i = 0; i < C::RM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(&A[(ty + C::TY * i) * C::LD + d]);
#pragma unroll
    for (int j = 0; j < C::RN; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(&Bm[(tx + 16 * j) * C::LD + d]);
#pragma unroll
    for (int i = 0; i < C::RM; ++i)
#pragma unroll
      for (int j = 0; j < C::RN; ++j) {
        acc2[i][j] = sm100::f2_fma(a[i].x, b[j].x, acc2[i][j]);
        acc2[i][j] = sm100::f2_fma(a[i].y, b[j].y, acc2[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < C::RM; ++i)
#pragma unroll
    for (int j = 0; j < C::RN; ++j) {
      float x, y;
      sm100::f2_unpack(acc2[i][j], x, y);
      acc[i][j] = x + y;
    }
}

// The block's values of one streamed column, for the thread's rows, next to each other (row ty + TY i in slot ty RM + i).
template <int D>
__device__ __forceinline__ void store_transposed(float* Xt, const float (&x)[Cfg<D>::RM][Cfg<D>::RN], int ty, int tx) {
  using C = Cfg<D>;
#pragma unroll
  for (int j = 0; j < C::RN; ++j) {
    float* dst = &Xt[(tx + 16 * j) * C::PLD + ty * C::RM];
    if (C::RM % 4 == 0) {
#pragma unroll
      for (int i = 0; i < C::RM; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(x[i][j], x[i + 1][j], x[i + 2][j], x[i + 3][j]);
    } else {
#pragma unroll
      for (int i = 0; i < C::RM; i += 2) *reinterpret_cast<float2*>(dst + i) = make_float2(x[i][j], x[i + 1][j]);
    }
  }
}

// acc[row pair][column] += sum_kk X[row][kk] * V[kk][column], X transposed in shared memory, V [kk][LD]
template <int D>
__device__ __forceinline__ void tile_xv(const float* Xt, const float* V, uint64_t (&acc)[Cfg<D>::RM / 2][Cfg<D>::DV], int ty, int tx) {
  using C = Cfg<D>;
#pragma unroll 4
  for (int kk = 0; kk < C::BN; ++kk) {
    uint64_t x[C::RM / 2];
    const float* xp = &Xt[kk * C::PLD + ty * C::RM];
    if (C::RM % 4 == 0) {
#pragma unroll
      for (int i = 0; i < C::RM / 4; ++i) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(xp + 4 * i);
        x[2 * i] = t.x;
        x[2 * i + 1] = t.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < C::RM / 2; ++i) x[i] = *reinterpret_cast<const uint64_t*>(xp + 2 * i);
    }
#pragma unroll
    for (int g = 0; g < C::NG; ++g) {
      float v[C::VEC];
      const float* vp = &V[kk * C::LD + g * 16 * C::VEC + tx * C::VEC];
      if (C::VEC == 4) {
        const float4 t = *reinterpret_cast<const float4*>(vp);
        v[0] = t.x, v[C::VEC > 1 ? 1 : 0] = t.y, v[C::VEC > 2 ? 2 : 0] = t.z, v[C::VEC > 3 ? 3 : 0] = t.w;
      } else if (C::VEC == 2) {
        const float2 t = *reinterpret_cast<const float2*>(vp);
        v[0] = t.x, v[C::VEC > 1 ? 1 : 0] = t.y;
      } else {
        v[0] = *vp;
      }
#pragma unroll
      for (int e = 0; e < C::VEC; ++e) {
        const uint64_t vv = sm100::f2_pack(v[e], v[e]);
#pragma unroll
        for (int i = 0; i < C::RM / 2; ++i) acc[i][g * C::VEC + e] = sm100::f2_fma(x[i], vv, acc[i][g * C::VEC + e]);
      }
    }
  }
}

template <int D>
__device__ __forceinline__ int col_of(int n, int tx) {  // head-dim column of a thread's n-th accumulator
  using C = Cfg<D>;
  return (n / C::VEC) * 16 * C::VEC + tx * C::VEC + n % C::VEC;
}

__device__ __forceinline__ float half_warp_max(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float half_warp_sum(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__device__ __forceinline__ int load_len(const int32_t* lens, int64_t stride, int b, int T_) {
  return lens ? kb_clamp_len(lens[(int64_t)b * stride], T_) : T_;
}

// The live keys of query i form the interval [lo, hi) (empty for a padded row): the element form of the mask.
__device__ __forceinline__ void live_interval(int i, int len, int c, int back, int& lo, int& hi) {
  lo = hi = 0;
  if (i < len) {
    const int qc = i / c;
    lo = kb_max_i32(0, qc - back) * c;
    const int64_t h = (int64_t)(qc + 1) * c;
    hi = h < len ? (int)h : len;
  }
}

// Rows of a thread's accumulators, scaled, into the contiguous [T, D] output slice; a column vector per store
// where the output is fp32 and aligned.
template <int D, typename T>
__device__ __forceinline__ void store_rows(T* slice, const uint64_t (&acc)[Cfg<D>::RM / 2][Cfg<D>::DV], const float (&scale)[Cfg<D>::RM],
                                           const bool (&zero)[Cfg<D>::RM], int row0, int T_, int ty, int tx) {
  using C = Cfg<D>;
  const bool vec = sizeof(T) == 4 && C::VEC == 4 && (reinterpret_cast<uintptr_t>(slice) & 15) == 0;
#pragma unroll
  for (int i = 0; i < C::RM; ++i) {
    const int r = row0 + ty + C::TY * i;
    if (r >= T_) continue;
    float x[C::DV];
#pragma unroll
    for (int n = 0; n < C::DV; ++n) {
      float a0, a1;
      sm100::f2_unpack(acc[i / 2][n], a0, a1);
      x[n] = zero[i] ? 0.f : (i & 1 ? a1 : a0) * scale[i];
    }
    T* dst = slice + (int64_t)r * D;
    if (vec) {
#pragma unroll
      for (int n = 0; n + 3 < C::DV; n += 4)
        *reinterpret_cast<float4*>(dst + col_of<D>(n, tx)) = make_float4(x[n], x[n + 1], x[n + 2], x[n + 3]);
    } else {
#pragma unroll
      for (int n = 0; n < C::DV; ++n) dst[col_of<D>(n, tx)] = from_f32<T>(x[n]);
    }
  }
}

// ------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------
template <int D, typename T>
__global__ void __launch_bounds__(Cfg<D>::kThreads, Cfg<D>::kCtasFwd) sa_fwd_generic_kernel(const FwdArgs<T> a) {
  using C = Cfg<D>;
  constexpr int BM = C::BM, BN = C::BN, RM = C::RM, RN = C::RN;
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;
  float* Ks = Qs + BM * C::LD;
  float* Vs = Ks + BN * C::LD;
  float* Pt = Vs + BN * C::LD;

  const int b = blockIdx.z, h = blockIdx.y, q0 = blockIdx.x * BM;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int T_ = a.T_, c = a.c, back = a.back;
  const int len = load_len(a.lens, a.lens_stride, b, T_);
  T* o_slice = a.o + ((int64_t)b * a.H + h) * T_ * D;
  float* lse_slice = a.lse ? a.lse + ((int64_t)b * a.H + h) * T_ : nullptr;

  const KbTileRange kr = kb_fwd_kv_range(q0, BM, BN, len, c, back);

  float m[RM], l[RM];
  int lo[RM], hi[RM];
  uint64_t acc[RM / 2][C::DV];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
    live_interval(q0 + ty + C::TY * i, len, c, back, lo[i], hi[i]);
  }
#pragma unroll
  for (int i = 0; i < RM / 2; ++i)
#pragma unroll
    for (int n = 0; n < C::DV; ++n) acc[i][n] = 0ull;

  if (kr.begin < kr.end) {
    load_tile<D, BM>(Qs, a.q, b, h, q0, T_);
    load_tile<D, BN>(Ks, a.k, b, h, kr.begin * BN, T_);
    load_tile<D, BN>(Vs, a.v, b, h, kr.begin * BN, T_);
    for (int kt = kr.begin; kt < kr.end; ++kt) {
      const int k0 = kt * BN;
      cp_async_wait<1>();  // everything but V
      __syncthreads();

      float s[RM][RN];
      tile_abt<D>(Qs, Ks, s, ty, tx);

#pragma unroll
      for (int i = 0; i < RM; ++i) {
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          const int kj = k0 + tx + 16 * j;
          s[i][j] = (kj >= lo[i] && kj < hi[i]) ? s[i][j] * a.scale_log2 : -INFINITY;
          mx = fmaxf(mx, s[i][j]);
        }
        mx = half_warp_max(mx);
        const float m_new = fmaxf(m[i], mx);
        const float m_safe = (m_new == -INFINITY) ? 0.f : m_new;
        const float alpha = exp2f(m[i] - m_safe);
        float rs = 0.f;
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          s[i][j] = exp2f(s[i][j] - m_safe);
          rs += s[i][j];
        }
        rs = half_warp_sum(rs);
        l[i] = l[i] * alpha + rs;
        m[i] = m_new;
#pragma unroll
        for (int n = 0; n < C::DV; ++n) {
          float a0, a1;
          sm100::f2_unpack(acc[i / 2][n], a0, a1);
          if (i & 1) a1 *= alpha; else a0 *= alpha;
          acc[i / 2][n] = sm100::f2_pack(a0, a1);
        }
      }
      store_transposed<D>(Pt, s, ty, tx);
      cp_async_wait<0>();
      __syncthreads();  // P and V are there, K has been read
      if (kt + 1 < kr.end) load_tile<D, BN>(Ks, a.k, b, h, k0 + BN, T_);
      tile_xv<D>(Pt, Vs, acc, ty, tx);
      __syncthreads();  // V and P have been read
      if (kt + 1 < kr.end) load_tile<D, BN>(Vs, a.v, b, h, k0 + BN, T_);
    }
  }

  float inv[RM];
  bool zero[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int r = q0 + ty + C::TY * i;
    zero[i] = r >= len;
    inv[i] = zero[i] ? 0.f : 1.f / l[i];
    if (lse_slice && tx == 0 && r < T_) lse_slice[r] = zero[i] ? 0.f : m[i] + log2f(l[i]);
  }
  store_rows<D, T>(o_slice, acc, inv, zero, q0, T_, ty, tx);
}

// ------------------------------------------------------------------------------------------
// backward, dQ pass (also produces delta = rowsum(O * dO))
// ------------------------------------------------------------------------------------------
template <int D, typename T>
__global__ void __launch_bounds__(Cfg<D>::kThreads, Cfg<D>::kCtasBwd) sa_bwd_dq_generic_kernel(const BwdArgs<T> a) {
  using C = Cfg<D>;
  constexpr int BM = C::BM, BN = C::BN, RM = C::RM, RN = C::RN;
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;
  float* dOs = Qs + BM * C::LD;
  float* Ks = dOs + BM * C::LD;
  float* Vs = Ks + BN * C::LD;
  float* dSt = Vs + BN * C::LD;

  const int b = blockIdx.z, h = blockIdx.y, q0 = blockIdx.x * BM;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int T_ = a.T_, c = a.c, back = a.back;
  const int len = load_len(a.lens, a.lens_stride, b, T_);
  const int64_t bh = (int64_t)b * a.H + h;
  T* dq_slice = a.dq + bh * T_ * D;
  float* delta_slice = a.delta + bh * T_;
  const float* lse_slice = a.lse + bh * T_;

  const KbTileRange kr = kb_fwd_kv_range(q0, BM, BN, len, c, back);

  uint64_t acc[RM / 2][C::DV];
  float delta[RM], lse[RM], scale[RM];
  bool zero[RM];
  int lo[RM], hi[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    delta[i] = 0.f;
    lse[i] = 0.f;
    scale[i] = a.sm_scale;
    zero[i] = false;
    live_interval(q0 + ty + C::TY * i, len, c, back, lo[i], hi[i]);
  }
#pragma unroll
  for (int i = 0; i < RM / 2; ++i)
#pragma unroll
    for (int n = 0; n < C::DV; ++n) acc[i][n] = 0ull;

  if (kr.begin < kr.end) {
    load_tile<D, BM>(Qs, a.q, b, h, q0, T_);
    load_tile<D, BM>(dOs, a.d_o, b, h, q0, T_);
    load_tile<D, BN>(Vs, a.v, b, h, kr.begin * BN, T_);
    load_tile<D, BN>(Ks, a.k, b, h, kr.begin * BN, T_);
    cp_async_wait<2>();  // Q and dO
    __syncthreads();
    const T* o_slice = a.o.p + b * a.o.sb + h * a.o.sh;
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const int r = q0 + ty + C::TY * i;
      float part = 0.f;
      if (r < len) {
#pragma unroll
        for (int n = 0; n < C::DV; ++n) {
          const int d = col_of<D>(n, tx);
          part = fmaf(to_f32(o_slice[(int64_t)r * a.o.st + (int64_t)d * a.o.sd]), dOs[(ty + C::TY * i) * C::LD + d], part);
        }
      }
      delta[i] = half_warp_sum(part);
      if (r < len) lse[i] = lse_slice[r];
    }

    for (int kt = kr.begin; kt < kr.end; ++kt) {
      const int k0 = kt * BN;
      cp_async_wait<0>();
      __syncthreads();

      float s[RM][RN], dp[RM][RN];
      tile_abt<D>(Qs, Ks, s, ty, tx);
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          const int kj = k0 + tx + 16 * j;
          s[i][j] = (kj >= lo[i] && kj < hi[i]) ? exp2f(s[i][j] * a.scale_log2 - lse[i]) : 0.f;
        }
      tile_abt<D>(dOs, Vs, dp, ty, tx);
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          const int kj = k0 + tx + 16 * j;
          s[i][j] = (kj >= lo[i] && kj < hi[i]) ? s[i][j] * (dp[i][j] - delta[i]) : 0.f;
        }
      store_transposed<D>(dSt, s, ty, tx);
      __syncthreads();  // dS is there, V has been read
      if (kt + 1 < kr.end) load_tile<D, BN>(Vs, a.v, b, h, k0 + BN, T_);
      tile_xv<D>(dSt, Ks, acc, ty, tx);
      __syncthreads();  // K and dS have been read
      if (kt + 1 < kr.end) load_tile<D, BN>(Ks, a.k, b, h, k0 + BN, T_);
    }
  }

  store_rows<D, T>(dq_slice, acc, scale, zero, q0, T_, ty, tx);
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int r = q0 + ty + C::TY * i;
    if (tx == 0 && r < T_) delta_slice[r] = delta[i];
  }
}

// ------------------------------------------------------------------------------------------
// backward, dK/dV pass (reads delta written by the dQ pass)
// ------------------------------------------------------------------------------------------
// SAVE: the dS tiles also go to the scratch, [query][key slot] as they lie in shared memory.
template <int D, typename T, bool SAVE>
__global__ void __launch_bounds__(Cfg<D>::kThreads, Cfg<D>::kCtasBwd) sa_bwd_dkdv_generic_kernel(const BwdArgs<T> a) {
  using C = Cfg<D>;
  constexpr int BM = C::BM, BN = C::BN, RM = C::RM, RN = C::RN;
  static_assert(BM == BN, "the score block is square: rows and columns swap roles here");
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;
  float* dOs = Qs + BM * C::LD;
  float* Ks = dOs + BM * C::LD;
  float* Vs = Ks + BN * C::LD;
  float* Pt = Vs + BN * C::LD;
  float* dSt = Pt + BM * C::PLD;
  float* lse_s = dSt + BM * C::PLD;
  float* delta_s = lse_s + BM;
  int* lo_s = reinterpret_cast<int*>(delta_s + BM);
  int* hi_s = lo_s + BM;

  const int b = blockIdx.z, h = blockIdx.y, k0 = blockIdx.x * BN;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int T_ = a.T_, c = a.c, back = a.back;
  const int len = load_len(a.lens, a.lens_stride, b, T_);
  const int64_t bh = (int64_t)b * a.H + h;
  T* dk_slice = a.dk + bh * T_ * D;
  T* dv_slice = a.dv + bh * T_ * D;
  const float* delta_slice = a.delta + bh * T_;
  const float* lse_slice = a.lse + bh * T_;

  const KbTileRange qr = kb_bwd_q_range(k0, BM, BN, len, c, back);

  // stationary rows are keys here, streamed columns are queries
  uint64_t acc_dk[RM / 2][C::DV], acc_dv[RM / 2][C::DV];
#pragma unroll
  for (int i = 0; i < RM / 2; ++i)
#pragma unroll
    for (int n = 0; n < C::DV; ++n) acc_dk[i][n] = acc_dv[i][n] = 0ull;

  if (qr.begin < qr.end) {
    load_tile<D, BN>(Ks, a.k, b, h, k0, T_);
    load_tile<D, BN>(Vs, a.v, b, h, k0, T_);
    for (int qt = qr.begin; qt < qr.end; ++qt) {
      const int q0 = qt * BM;
      load_tile<D, BM>(Qs, a.q, b, h, q0, T_);
      load_tile<D, BM>(dOs, a.d_o, b, h, q0, T_);
      if (threadIdx.x < BM) {
        const int r = q0 + threadIdx.x;
        lse_s[threadIdx.x] = r < len ? lse_slice[r] : 0.f;
        delta_s[threadIdx.x] = r < len ? delta_slice[r] : 0.f;
        live_interval(r, len, c, back, lo_s[threadIdx.x], hi_s[threadIdx.x]);
      }
      cp_async_wait<0>();
      __syncthreads();

      float s[RM][RN], dp[RM][RN];
      tile_abt<D>(Ks, Qs, s, ty, tx);
#pragma unroll
      for (int j = 0; j < RN; ++j) {
        const int lo = lo_s[tx + 16 * j], hi = hi_s[tx + 16 * j];
        const float lse = lse_s[tx + 16 * j];
#pragma unroll
        for (int i = 0; i < RM; ++i) {
          const int kj = k0 + ty + C::TY * i;
          s[i][j] = (kj >= lo && kj < hi) ? exp2f(s[i][j] * a.scale_log2 - lse) : 0.f;
        }
      }
      store_transposed<D>(Pt, s, ty, tx);
      tile_abt<D>(Vs, dOs, dp, ty, tx);
#pragma unroll
      for (int j = 0; j < RN; ++j) {
        const int lo = lo_s[tx + 16 * j], hi = hi_s[tx + 16 * j];
        const float delta = delta_s[tx + 16 * j];
#pragma unroll
        for (int i = 0; i < RM; ++i) {
          const int kj = k0 + ty + C::TY * i;
          s[i][j] = (kj >= lo && kj < hi) ? s[i][j] * (dp[i][j] - delta) : 0.f;
        }
      }
      store_transposed<D>(dSt, s, ty, tx);
      __syncthreads();
      if (SAVE) {
        float4* dst = reinterpret_cast<float4*>(ds_tile<D, T>(a, bh, blockIdx.x, qt - qr.begin));
        for (int idx = threadIdx.x; idx < BM * BN / 4; idx += C::kThreads) {
          const int r = idx / (BN / 4), k4 = (idx - r * (BN / 4)) * 4;
          dst[idx] = *reinterpret_cast<const float4*>(&dSt[r * C::PLD + k4]);
        }
      }
      tile_xv<D>(Pt, dOs, acc_dv, ty, tx);
      tile_xv<D>(dSt, Qs, acc_dk, ty, tx);
      __syncthreads();
    }
  }

  float sc_k[RM], sc_v[RM];
  bool zero[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    sc_k[i] = a.sm_scale;
    sc_v[i] = 1.f;
    zero[i] = false;
  }
  store_rows<D, T>(dk_slice, acc_dk, sc_k, zero, k0, T_, ty, tx);
  store_rows<D, T>(dv_slice, acc_dv, sc_v, zero, k0, T_, ty, tx);
}

// ------------------------------------------------------------------------------------------
// backward with the scores evaluated once (fp32): delta, then dK/dV saving dS, then dQ = dS K
// ------------------------------------------------------------------------------------------
// Sixteen lanes per row with the columns the dQ pass gives them, so that delta has the same bits.
template <int D, typename T>
__global__ void __launch_bounds__(256) sa_bwd_delta_generic_kernel(const BwdArgs<T> a) {
  using C = Cfg<D>;
  const int b = blockIdx.z, h = blockIdx.y, tx = threadIdx.x & 15;
  const int len = load_len(a.lens, a.lens_stride, b, a.T_);
  const T* o_slice = a.o.p + b * a.o.sb + h * a.o.sh;
  const T* g_slice = a.d_o.p + b * a.d_o.sb + h * a.d_o.sh;
#pragma unroll
  for (int it = 0; it < C::BM / 16; ++it) {
    const int r = blockIdx.x * C::BM + it * 16 + (threadIdx.x >> 4);
    float part = 0.f;
    if (r < len) {
#pragma unroll
      for (int n = 0; n < C::DV; ++n) {
        const int64_t d = col_of<D>(n, tx);
        part = fmaf(to_f32(o_slice[(int64_t)r * a.o.st + d * a.o.sd]), to_f32(g_slice[(int64_t)r * a.d_o.st + d * a.d_o.sd]), part);
      }
    }
    part = half_warp_sum(part);
    if (tx == 0 && r < a.T_) a.delta[((int64_t)b * a.H + h) * a.T_ + r] = part;
  }
}

// One CTA per query tile: streams the saved dS tiles of its key tiles with the matching K tiles.  A third of the
// dQ pass's arithmetic for one write and one read of 4 bytes per score (202 -> 65 us, dK/dV pass 260 -> 264).  Small
// CTAs with single buffers: five or more on an SM cover each other's loads.
template <int D, typename T>
__global__ void __launch_bounds__(Cfg<D>::kThreads) sa_bwd_dq_saved_generic_kernel(const BwdArgs<T> a) {
  using C = Cfg<D>;
  constexpr int BM = C::BM, BN = C::BN, RM = C::RM, SLD = BN + kPad;
  extern __shared__ __align__(16) float smem[];
  float* Ss = smem;  // dS tile, [query][key slot]
  float* Ks = Ss + BM * SLD;

  const int b = blockIdx.z, h = blockIdx.y, qt = blockIdx.x, q0 = qt * BM;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int T_ = a.T_;
  const int len = load_len(a.lens, a.lens_stride, b, T_);
  const int64_t bh = (int64_t)b * a.H + h;
  const KbTileRange kr = kb_fwd_kv_range(q0, BM, BN, len, a.c, a.back);

  float acc[RM][C::DV];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int n = 0; n < C::DV; ++n) acc[i][n] = 0.f;

  for (int kt = kr.begin; kt < kr.end; ++kt) {
    // the slot this query tile has in key tile kt's list: both schedules name the same pairs
    const KbTileRange qr = kb_bwd_q_range(kt * BN, BM, BN, len, a.c, a.back);
    const float* src = ds_tile<D, T>(a, bh, kt, qt - qr.begin);
    for (int idx = threadIdx.x; idx < BM * BN / 4; idx += C::kThreads) {
      const int r = idx / (BN / 4), k4 = (idx - r * (BN / 4)) * 4;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm100::smem_u32(Ss + r * SLD + k4)), "l"(src + idx * 4) : "memory");
    }
    load_tile<D, BN>(Ks, a.k, b, h, kt * BN, T_);
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll 2
    for (int s4 = 0; s4 < BN; s4 += 4) {
      float4 x[RM];
#pragma unroll
      for (int i = 0; i < RM; ++i) x[i] = *reinterpret_cast<const float4*>(&Ss[(ty + C::TY * i) * SLD + s4]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int slot = s4 + e, key = slot / RM + C::TY * (slot % RM);  // see store_transposed
        float k[C::DV];
#pragma unroll
        for (int n = 0; n < C::DV; n += C::VEC) {
          const float* kp = &Ks[key * C::LD + col_of<D>(n, tx)];
          if constexpr (C::VEC == 4) {
            const float4 t = *reinterpret_cast<const float4*>(kp);
            k[n] = t.x, k[n + 1] = t.y, k[n + 2] = t.z, k[n + 3] = t.w;
          } else {
#pragma unroll
            for (int v = 0; v < C::VEC; ++v) k[n + v] = kp[v];
          }
        }
#pragma unroll
        for (int i = 0; i < RM; ++i) {
          const float xv = e == 0 ? x[i].x : e == 1 ? x[i].y : e == 2 ? x[i].z : x[i].w;
#pragma unroll
          for (int n = 0; n < C::DV; ++n) acc[i][n] = fmaf(xv, k[n], acc[i][n]);
        }
      }
    }
    __syncthreads();
  }

  uint64_t out[RM / 2][C::DV];
  float scale[RM];
  bool zero[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    scale[i] = a.sm_scale;
    zero[i] = false;
#pragma unroll
    for (int n = 0; n < C::DV; ++n)
      if (i % 2 == 0) out[i / 2][n] = sm100::f2_pack(acc[i][n], acc[i + 1][n]);
  }
  store_rows<D, T>(a.dq + bh * T_ * D, out, scale, zero, q0, T_, ty, tx);
}

// ------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------
template <int D, typename T>
int launch_fwd(const kb_sa_fwd_params& p, int32_t c, int32_t back, cudaStream_t s) {
  using C = Cfg<D>;
  constexpr size_t smem = sizeof(float) * (size_t)(C::BM * C::LD + 2 * C::BN * C::LD + C::BN * C::PLD);
  auto kern = sa_fwd_generic_kernel<D, T>;
  int dev = 0, n_sm = 0;
  if (!device_sm_count(&dev, &n_sm)) return KB_ERR_LAUNCH;
  static std::atomic<bool> smem_opted_in[kMaxDevices];
  KB_CUDA_TRY(opt_in_smem_once(kern, smem, dev, smem_opted_in));
  FwdArgs<T> a;
  a.q = make_arg<T>(p.q);
  a.k = make_arg<T>(p.k);
  a.v = make_arg<T>(p.v);
  a.o = static_cast<T*>(p.o);
  a.lse = p.lse;
  a.lens = p.lens;
  a.lens_stride = p.lens_stride;
  a.H = p.H;
  a.T_ = p.T;
  a.c = c;
  a.back = back;
  a.scale_log2 = p.sm_scale * kLog2e;
  dim3 grid(kb_cdiv_i32(p.T, C::BM), p.H, p.B);
  kern<<<grid, C::kThreads, smem, s>>>(a);
  KB_LAUNCH_CHECK("sa_fwd_generic_kernel");
  return KB_OK;
}

template <int D, typename T>
int launch_bwd(const kb_sa_bwd_params& p, int32_t c, int32_t back, cudaStream_t s) {
  using C = Cfg<D>;
  constexpr size_t smem_dq = sizeof(float) * (size_t)(2 * C::BM * C::LD + 2 * C::BN * C::LD + C::BN * C::PLD);
  constexpr size_t smem_dkdv = sizeof(float) * (size_t)(2 * C::BM * C::LD + 2 * C::BN * C::LD + 2 * C::BM * C::PLD + 4 * C::BM);
  static_assert(smem_dkdv <= 232448, "shared memory exceeds the 227 KB a CTA may have");
  auto kern_dq = sa_bwd_dq_generic_kernel<D, T>;
  auto kern_dkdv = sa_bwd_dkdv_generic_kernel<D, T, false>;
  int dev = 0, n_sm = 0;
  if (!device_sm_count(&dev, &n_sm)) return KB_ERR_LAUNCH;
  static std::atomic<bool> dq_opted_in[kMaxDevices], dkdv_opted_in[kMaxDevices];
  KB_CUDA_TRY(opt_in_smem_once(kern_dq, smem_dq, dev, dq_opted_in));
  KB_CUDA_TRY(opt_in_smem_once(kern_dkdv, smem_dkdv, dev, dkdv_opted_in));
  BwdArgs<T> a;
  a.q = make_arg<T>(p.q);
  a.k = make_arg<T>(p.k);
  a.v = make_arg<T>(p.v);
  a.o = make_arg<T>(p.o);
  a.d_o = make_arg<T>(p.d_o);
  a.lse = p.lse;
  a.dq = static_cast<T*>(p.dq);
  a.dk = static_cast<T*>(p.dk);
  a.dv = static_cast<T*>(p.dv);
  a.delta = p.delta_ws;
  a.ds = nullptr;
  a.W = 0;
  a.lens = p.lens;
  a.lens_stride = p.lens_stride;
  a.H = p.H;
  a.T_ = p.T;
  a.c = c;
  a.back = back;
  a.scale_log2 = p.sm_scale * kLog2e;
  a.sm_scale = p.sm_scale;
  dim3 grid_q(kb_cdiv_i32(p.T, C::BM), p.H, p.B), grid_k(kb_cdiv_i32(p.T, C::BN), p.H, p.B);
  if constexpr (sizeof(T) == 4) {
    // Scores evaluated once where the caller gives the scratch (and asks for no single pass): three launches, 14 instead
    // of 18 multiplications per pair and head-dim element over forward and backward.
    const uint32_t passes = KB_FLAG_BWD_SKIP_DQ | KB_FLAG_BWD_SKIP_DKDV | KB_FLAG_BWD_SKIP_DELTA | KB_FLAG_BWD_TWO_PASS;
    if (p.ds_ws && !(p.flags & passes) && reinterpret_cast<uintptr_t>(p.ds_ws) % 16 == 0 &&
        p.ds_ws_bytes >= sa_bwd_generic_workspace_bytes(p.B, p.H, p.T, D, c, back)) {
      constexpr size_t smem_saved = sizeof(float) * (size_t)(C::BM * (C::BN + kPad) + C::BN * C::LD);
      auto kern_save = sa_bwd_dkdv_generic_kernel<D, T, true>;
      auto kern_saved = sa_bwd_dq_saved_generic_kernel<D, T>;
      static std::atomic<bool> save_opted_in[kMaxDevices], saved_opted_in[kMaxDevices];
      KB_CUDA_TRY(opt_in_smem_once(kern_save, smem_dkdv, dev, save_opted_in));
      KB_CUDA_TRY(opt_in_smem_once(kern_saved, smem_saved, dev, saved_opted_in));
      a.ds = static_cast<float*>(p.ds_ws);
      a.W = ds_slots(p.T, C::BM, c, back);
      sa_bwd_delta_generic_kernel<D, T><<<grid_q, 256, 0, s>>>(a);
      KB_LAUNCH_CHECK("sa_bwd_delta_generic_kernel");
      kern_save<<<grid_k, C::kThreads, smem_dkdv, s>>>(a);
      KB_LAUNCH_CHECK("sa_bwd_dkdv_generic_kernel");
      kern_saved<<<grid_q, C::kThreads, smem_saved, s>>>(a);
      KB_LAUNCH_CHECK("sa_bwd_dq_saved_generic_kernel");
      return KB_OK;
    }
  }
  if (!(p.flags & KB_FLAG_BWD_SKIP_DQ)) {
    kern_dq<<<grid_q, C::kThreads, smem_dq, s>>>(a);
    KB_LAUNCH_CHECK("sa_bwd_dq_generic_kernel");
  }
  if (!(p.flags & KB_FLAG_BWD_SKIP_DKDV)) {
    kern_dkdv<<<grid_k, C::kThreads, smem_dkdv, s>>>(a);
    KB_LAUNCH_CHECK("sa_bwd_dkdv_generic_kernel");
  }
  return KB_OK;
}

template <typename T, typename P, typename F>
int dispatch_head_dim(const P& p, F&& f) {
  switch (p.D) {
    case 16: return f(std::integral_constant<int, 16>{});
    case 32: return f(std::integral_constant<int, 32>{});
    case 64: return f(std::integral_constant<int, 64>{});
    case 128: return f(std::integral_constant<int, 128>{});
    case 256: return f(std::integral_constant<int, 256>{});
    default: return KB_ERR_UNSUPPORTED;
  }
}

}  // namespace

int sa_fwd_generic(const kb_sa_fwd_params& p, int32_t c, int32_t back, cudaStream_t s) {
  switch (p.dtype) {
    case KB_F32:
      return dispatch_head_dim<float>(p, [&](auto d) { return launch_fwd<decltype(d)::value, float>(p, c, back, s); });
    case KB_F16:
      return dispatch_head_dim<__half>(p, [&](auto d) { return launch_fwd<decltype(d)::value, __half>(p, c, back, s); });
    case KB_BF16:
      return dispatch_head_dim<__nv_bfloat16>(
          p, [&](auto d) { return launch_fwd<decltype(d)::value, __nv_bfloat16>(p, c, back, s); });
    default:
      return KB_ERR_UNSUPPORTED;
  }
}

// Bytes of dS scratch the single-evaluation fp32 backward needs; c and back already clamped to T.
size_t sa_bwd_generic_workspace_bytes(int32_t B, int32_t H, int32_t T, int32_t D, int32_t c, int32_t back) {
  const int32_t tile = tiles::generic_tile(D);
  return (size_t)B * H * kb_cdiv_i32(T, tile) * ds_slots(T, tile, c, back) * tile * tile * sizeof(float);
}

int sa_bwd_generic(const kb_sa_bwd_params& p, int32_t c, int32_t back, cudaStream_t s) {
  switch (p.dtype) {
    case KB_F32:
      return dispatch_head_dim<float>(p, [&](auto d) { return launch_bwd<decltype(d)::value, float>(p, c, back, s); });
    case KB_F16:
      return dispatch_head_dim<__half>(p, [&](auto d) { return launch_bwd<decltype(d)::value, __half>(p, c, back, s); });
    case KB_BF16:
      return dispatch_head_dim<__nv_bfloat16>(
          p, [&](auto d) { return launch_bwd<decltype(d)::value, __nv_bfloat16>(p, c, back, s); });
    default:
      return KB_ERR_UNSUPPORTED;
  }
}

}  // namespace kb
