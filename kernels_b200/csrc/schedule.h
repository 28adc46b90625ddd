// Tile schedule of streaming attention: which KV tiles a q tile visits and which q tiles a
// KV tile receives gradient from.  One definition shared by the host planner (kb_sa_plan)
// and every kernel, so the schedule the tests check bit-exactly is the one the GPU walks.
//
// Mask: (i, j) is live iff  i < len, j < len and 0 <= i/c - j/c <= back
// (reference: src/streaming_attention/kernel.py:1540-1551).
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define KB_HD __host__ __device__ __forceinline__
#else
#define KB_HD inline
#endif

struct KbTileRange {
  int32_t begin;
  int32_t end;  // one past the last tile; begin == end means nothing to visit
};

KB_HD int32_t kb_min_i32(int32_t a, int32_t b) { return a < b ? a : b; }
KB_HD int32_t kb_max_i32(int32_t a, int32_t b) { return a > b ? a : b; }
KB_HD int32_t kb_cdiv_i32(int32_t a, int32_t b) { return (a + b - 1) / b; }

// Clamp of the user's length to [0, T] (kernel.py:238-239) and of the chunk parameters to
// ranges in which all later products stay inside int32: a chunk longer than the sequence
// is one chunk, and looking back further than the number of chunks changes nothing.
KB_HD int32_t kb_clamp_len(int64_t len, int32_t T) { return len < 0 ? 0 : (len > T ? T : (int32_t)len); }
KB_HD int32_t kb_clamp_context(int64_t c, int32_t T) { return c > T ? kb_max_i32(T, 1) : (int32_t)c; }
KB_HD int32_t kb_clamp_back(int64_t back, int32_t T, int32_t c) {
  int32_t n = kb_cdiv_i32(kb_max_i32(T, 1), c);
  return back > n ? n : (int32_t)back;
}

// KV tiles visited by the q tile that starts at token q0 (kernel.py:243-244, 282-291).
KB_HD KbTileRange kb_fwd_kv_range(int32_t q0, int32_t tile_q, int32_t tile_k, int32_t len, int32_t c,
                                  int32_t back) {
  KbTileRange r = {0, 0};
  if (len <= q0) return r;
  int32_t min_ctx = q0 / c;
  r.begin = kb_max_i32(0, (min_ctx - back) * c) / tile_k;
  int32_t q_hi = kb_min_i32(q0 + tile_q, len);
  int32_t max_ctx = (q_hi - 1) / c;
  // (max_ctx + 1) * c can exceed int32 only if it exceeds len; compare in 64 bit.
  int64_t hi = (int64_t)(max_ctx + 1) * c;
  r.end = kb_cdiv_i32(hi < len ? (int32_t)hi : len, tile_k);
  return r;
}

// q tiles that send gradient to the KV tile starting at token k0 (kernel.py:1046-1054).
KB_HD KbTileRange kb_bwd_q_range(int32_t k0, int32_t tile_q, int32_t tile_k, int32_t len, int32_t c,
                                 int32_t back) {
  KbTileRange r = {0, 0};
  if (len <= k0) return r;
  int32_t min_ctx = k0 / c;
  r.begin = (min_ctx * c) / tile_q;
  int32_t k_max_tok = kb_min_i32(k0 + tile_k, len) - 1;
  int32_t max_ctx = k_max_tok / c;
  int64_t hi = (int64_t)(max_ctx + back + 1) * c;
  r.end = kb_cdiv_i32(hi < len ? (int32_t)hi : len, tile_q);
  return r;
}

// Division of a non-negative int32 by a positive int32 that is fixed for a launch, as one
// multiply-high, add and shift instead of the ~100-cycle integer-division sequence: the
// persistent kernels decode a work item (several divisions by the head count, the tile count
// and the chunk length) on their critical path every few tiles.  Exact for 0 <= n < 2^31.
struct KbFastDiv {
  uint32_t mul, shift, d;
};
inline KbFastDiv kb_fastdiv_make(int32_t divisor) {
  KbFastDiv f;
  f.d = (uint32_t)(divisor < 1 ? 1 : divisor);
  uint32_t s = 0;
  while (((uint64_t)1 << s) < f.d) ++s;  // s = ceil(log2 d)
  f.shift = s;
  f.mul = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << s) - f.d)) / f.d + 1);
  return f;
}
KB_HD int32_t kb_fastdiv(int32_t n, const KbFastDiv& f) {
#if defined(__CUDA_ARCH__)
  const uint32_t hi = __umulhi((uint32_t)n, f.mul);
#else
  const uint32_t hi = (uint32_t)(((uint64_t)(uint32_t)n * f.mul) >> 32);
#endif
  return (int32_t)((hi + (uint32_t)n) >> f.shift);
}

// The order in which the CTAs of the main backward kernel take the work items (the others take them as they become free,
// item_queue.cuh).  Wave w hands out the items
// [w G, (w + 1) G) (G = CTAs): neighbouring items run at the same time and share their K / V rows in L2.  Inside a
// wave CTA x takes number (x + w r) mod G.  An item's place in its sequence is item mod n (n = items per sequence and
// head); with r = 0 a CTA meets only n / gcd(G, n) of the places.  Where sequences differ in length the late places are
// often padding, and with few places per CTA some CTAs get much more work than others (n = 4, G = 148: CTA 0 only the
// first quarter of every sequence).  r > 0 makes G + r and n coprime, which spreads the places.
//
// Only where the lengths differ and a CTA would meet at most `most_places` places (1 to 4).  Measured (B200, r = 0 / r = 1):
// packed batch of 256 sequences of 128-1024 rows 1286 / 1081 us.  With eight and more places nothing is gained, and
// an odd r can cost: bf16 D=128 c=256 T=16384: 1680 us with even r, 1890-1980 with odd r (with an even one
// CTAs 2 m and 2 m + 1 always have the two key tiles of one chunk, which stream the same Q / dO tiles).
//
// Chunks that are whole pairs of key tiles (c a multiple of 256) are therefore shifted only where a
// CTA meets fewer places than four.  r = 0 / shifted, us, bf16 D=128, by the places met: padded, lengths T/2 to T: one (T=512)
// 782 / 818; two (T=1024) 909 / 977, four (T=2048) 954 / 1035; c=512 T=768 (three) 928 / 1006.  Packed, T/8 to T:
// one 1390 / 1145, two 1369 / 1340, four 1400 / 1470.  fp16 D=64 c=256, padded: one 334 / 289, two 409 / 385, four 451 /
// 464.  Hence at most two, at most one for the padded head-dim-128 class.  (Other chunk lengths gain everywhere, but for
// c=160 and 192 at T=512: 784 / 834.)
inline int32_t kb_gcd(int32_t a, int32_t b) {
  while (b) {
    const int32_t t = a % b;
    a = b;
    b = t;
  }
  return a;
}
inline int32_t kb_item_rotation(int32_t ctas, int32_t items_per_seq, bool ragged, int32_t most_places = 4) {
  const int32_t n = items_per_seq;
  if (!ragged || ctas < 1 || n < 1 || n / kb_gcd(ctas, n) > most_places) return 0;
  int32_t r = 0;
  while (kb_gcd(ctas + r, n) != 1) ++r;  // among n consecutive numbers one is coprime to n
  return r % ctas;
}
#if defined(__CUDACC__)
struct KbItemWalk {
  int32_t base, off, rot;
  __device__ __forceinline__ explicit KbItemWalk(int32_t rotation) : base(0), off((int32_t)blockIdx.x), rot(rotation) {}
  __device__ __forceinline__ int32_t item() const { return base + off; }  // the walk ends at the first item() >= n_items
  __device__ __forceinline__ void next() {
    base += (int32_t)gridDim.x;
    off += rot;
    if (off >= (int32_t)gridDim.x) off -= (int32_t)gridDim.x;
  }
};
#endif

// The two tile ranges above with the divisions by the chunk length done by kb_fastdiv (same
// results; the persistent kernels call these).
KB_HD KbTileRange kb_fwd_kv_range_fd(int32_t q0, int32_t tile_q, int32_t tile_k, int32_t len, int32_t c,
                                     int32_t back, const KbFastDiv& fc) {
  KbTileRange r = {0, 0};
  if (len <= q0) return r;
  int32_t min_ctx = kb_fastdiv(q0, fc);
  r.begin = kb_max_i32(0, (min_ctx - back) * c) / tile_k;
  int32_t q_hi = kb_min_i32(q0 + tile_q, len);
  int32_t max_ctx = kb_fastdiv(q_hi - 1, fc);
  int64_t hi = (int64_t)(max_ctx + 1) * c;
  r.end = kb_cdiv_i32(hi < len ? (int32_t)hi : len, tile_k);
  return r;
}
KB_HD KbTileRange kb_bwd_q_range_fd(int32_t k0, int32_t tile_q, int32_t tile_k, int32_t len, int32_t c,
                                    int32_t back, const KbFastDiv& fc) {
  KbTileRange r = {0, 0};
  if (len <= k0) return r;
  int32_t min_ctx = kb_fastdiv(k0, fc);
  r.begin = (min_ctx * c) / tile_q;
  int32_t k_max_tok = kb_min_i32(k0 + tile_k, len) - 1;
  int32_t max_ctx = kb_fastdiv(k_max_tok, fc);
  int64_t hi = (int64_t)(max_ctx + back + 1) * c;
  r.end = kb_cdiv_i32(hi < len ? (int32_t)hi : len, tile_q);
  return r;
}

// Element mask.  qc / kc are the chunk indices i/c and j/c.
KB_HD bool kb_live(int32_t i, int32_t j, int32_t qc, int32_t kc, int32_t len, int32_t back) {
  int32_t diff = qc - kc;
  return i < len && j < len && diff >= 0 && diff <= back;
}
