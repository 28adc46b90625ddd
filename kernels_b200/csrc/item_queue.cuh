// The work items of the persistent kernels, handed out while the kernel runs.
//
// The grid has one block per work item, one block fits an SM, and a running CTA takes over blocks that have not been
// launched yet (clusterlaunchcontrol.try_cancel): it starts with the item of its own block index and asks for another
// when it is about to run out.  So a CTA that meets padding or short items simply comes back sooner.  No counter in
// global memory: nothing to clear before a launch, nothing that calls, streams or graph replays could share.
//
// One warp of the CTA, the TMA producer's, asks (ItemWriter).  It clears the outputs of items that lie wholly in the
// padding itself and passes the live ones to the other roles through a ring of kItemSlots numbers in shared memory
// (ItemReader).  (Padded items do not go through the ring: a role may look for the next live item before the current one
// is complete, and would wait for ever behind a run of padded ones that fills the ring.)  It asks when it has
// issued the loads of an item's last tiles: the answer takes 350 clocks, and an item claimed earlier would wait at a CTA that is still busy.
// Or (n_fixed) it takes the items in turn with the grid's other CTAs; sa_bwd_fused_sm100.cu says where that is better.
//
// A block without work costs that answer all the same, so a packed batch does not launch a block for every tile of its
// longest sequence times every sequence where that is mostly padding (PackedGrid).
#pragma once
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace kb {
namespace sm100 {

constexpr int kItemSlots = 4;
constexpr int kItemsOver = -1, kItemPadding = -2;
enum ItemWaitSite { kWaitItemAnswer = 121, kWaitItemEmpty, kWaitItemFull };

struct alignas(16) ItemQueue {
  uint32_t answer[4];
  int4 entry[kItemSlots];  // item (-1: there are no more), and what its writer says about it
  uint64_t answered, full[kItemSlots], empty[kItemSlots];
};

// `readers`: ItemReaders of the CTA.  Executed by one thread, before fence_mbar_init() and the CTA's first barrier.
__device__ __forceinline__ void item_queue_init(ItemQueue& q, int readers) {
  mbar_init(&q.answered, 1);
  for (int i = 0; i < kItemSlots; ++i) {
    mbar_init(&q.full[i], 1);
    mbar_init(&q.empty[i], readers);
  }
}

__device__ __forceinline__ void item_ask(ItemQueue* q) {
  mbar_expect_tx(&q->answered, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   smem_u32(q->answer)),
               "r"(smem_u32(&q->answered))
               : "memory");
}
// The block index in the answer, kItemsOver if there was no block left to take over (after which none may be asked for).
__device__ __forceinline__ int item_answer(const ItemQueue* q) {
  uint32_t got, x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 a;\n\t.reg .b32 y, z, w;\n\t"
      "ld.shared.b128 a, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n\t"
      "selp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, y, z, w}, a;\n\t}"
      : "=r"(got), "=&r"(x)
      : "r"(smem_u32(q->answer))
      : "memory");
  fence_proxy_async();  // (the next answer is written through the async proxy)
  return got ? (int)x : kItemsOver;
}
// After a wait of the CTA gave up: the blocks not launched yet are taken over and dropped, so that the kernel ends with
// the error code now and not after as many such waits as there are items left.  `answers`: answers taken so far.
static __device__ __noinline__ void item_drop_rest(ItemQueue* q, int answers, bool asked) {
  for (int item = 0; item >= 0; ++answers) {
    if (!asked) item_ask(q);
    asked = false;
    for (uint32_t spins = 0; !mbar_try_wait(&q->answered, answers & 1);)
      if (++spins >= kWaitLimitSpins) return;
    item = item_answer(q);
  }
}

// The blocks of a packed batch, [sequence][head][tile of the sequence]: sequence b begins at block heads * (cu[b] / tile +
// b).  That leaves every (sequence, head) room for its own tiles and at most one more, and needs nothing of the lengths but
// their sum on the host and their offsets here.  With a block per tile of the longest sequence (n_seqs = 0, item = block)
// one sequence of 32 768 rows among 1 000 of 100 (16 heads, D = 128, c = 64) has 4.1 M blocks in the main kernel, of which
// 20 thousand have work.  Block per tile / this, us: forward 6 700 / 626, main 14 330 / 812, dQ 12 520 / 397; 16 384 among
// 500 of 60 (8 heads, D = 64) 880 / 124, 1 850 / 177, 1 614 / 87.  Finding a block's item takes the loads of two searches
// and two divisions, which batches of short items notice; so the host takes this grid where it has less than half as many
// blocks: at 0.44 of them (2 048 rows and four of 448, forty times) forward 525 / 529, main 930 / 942, dQ 368 / 353.
struct PackedGrid {
  const int32_t* cu;
  int32_t n_seqs, heads, shift, T, n_tiles;  // tiles of 2^shift rows; T: the longest sequence, n_tiles: its tiles
};
// The item of a block, as (sequence * heads + head) * n_tiles + tile, kItemPadding if it has none.  By a whole warp: 32
// sequences are looked at at a time.  Out of line: in the main kernel's loop it cost every packed batch 3 to 5 %.
static __device__ __noinline__ int packed_item(const int32_t* cu, int n_seqs, int heads, int shift, int T, int n_tiles, int block) {
  const int lane = threadIdx.x & 31;
  int b = 0;
  for (int n = n_seqs; n > 1;) {  // the block belongs to one of the sequences [b, b + n)
    const int step = (n + 31) >> 5, at = lane * step;
    const bool begun = at < n && heads * ((cu[b + at] >> shift) + b + at) <= block;
    const int skip = kb_max_i32(__popc(__ballot_sync(0xffffffffu, begun)) - 1, 0) * step;
    b += skip;
    n = kb_min_i32(step, n - skip);
  }
  const int row0 = cu[b], end = cu[b + 1];
  const int per_head = kb_max_i32((end >> shift) - (row0 >> shift) + 1, 1);
  const int rest = block - heads * ((row0 >> shift) + b);
  const int h = rest / per_head, tile = rest - h * per_head;
  if (rest < 0 || h >= heads || tile << shift >= kb_min_i32(end - row0, T)) return kItemPadding;
  return (b * heads + h) * n_tiles + tile;
}
// ... and on the host: the number of blocks of a packed batch, and which of the two grids they are.
inline int64_t packed_grid_blocks(PackedGrid& g, const int32_t* cu, int32_t B, int32_t heads, int32_t T, int32_t total, int32_t shift) {
  const int32_t n_tiles = kb_cdiv_i32(T, 1 << shift);
  const int64_t each = (int64_t)B * heads * n_tiles, own = (int64_t)heads * ((total >> shift) + B);
  const bool by_rows = 2 * own < each;
  g = PackedGrid{cu, by_rows ? B : 0, heads, shift, T, n_tiles};
  return by_rows ? own : each;
}

// Used by a whole converged warp; item() is the same in all lanes, the rest is lane 0's.
template <bool PACKED>
struct ItemWriter {
  ItemQueue* q;
  const PackedGrid& grid;         // (in the kernel's parameters; used if PACKED)
  int n_fixed;                    // > 0: the CTAs of the grid take these items in turn, nothing is asked for
  int answers, published, item_;  // answers taken, items passed on so far; the current item, kItemsOver after the last one
  bool asked, more, ok;          // a request is under way; no request has failed yet; no wait gave up
  __device__ __forceinline__ ItemWriter(ItemQueue& queue, const PackedGrid& packed_grid, int fixed = 0)
      : q(&queue), grid(packed_grid), n_fixed(fixed), answers(0), published(0), item_(of_block((int)blockIdx.x)), asked(false), more(fixed == 0), ok(true) {}
  __device__ __forceinline__ bool more_items() const { return PACKED ? item_ != kItemsOver : item_ >= 0; }
  __device__ __forceinline__ int of_block(int block) const {
    if (!PACKED || grid.n_seqs == 0 || block < 0) return block;
    return packed_item(grid.cu, grid.n_seqs, grid.heads, grid.shift, grid.T, grid.n_tiles, block);
  }
  __device__ __forceinline__ int item() const { return item_; }
  // Lane 0: ask for the next item ahead of next().
  __device__ __forceinline__ void ask() {
    if (!asked && n_fixed == 0) item_ask(q);
    asked = true;
  }
  // Lane 0: pass an item on to the readers.
  __device__ __forceinline__ bool publish(int4 entry, const WaitCtx& ctx) {
    const int n = published++, s = n % kItemSlots;
    if (n >= kItemSlots && !mbar_wait(&q->empty[s], ((n / kItemSlots) - 1) & 1, ctx, kWaitItemEmpty)) return false;
    q->entry[s] = entry;
    mbar_arrive(&q->full[s]);
    return true;
  }
  // The warp's next item; `go_on` (lane 0's counts): false ends the walk after an error.
  __device__ __forceinline__ void next(bool go_on, const WaitCtx& ctx) {
    int got = -1;
    if ((threadIdx.x & 31) == 0) {
      ok = go_on;
      if (ok && n_fixed > 0) {
        got = item_ + (int)gridDim.x;
        if (got >= n_fixed) got = -1;
      } else if (ok) {
        ask();
        ok = mbar_wait(&q->answered, answers & 1, ctx, kWaitItemAnswer);
        if (ok) {
          asked = false;
          ++answers;
          got = item_answer(q);
          more = got >= 0;
        }
      }
    }
    item_ = of_block(__shfl_sync(0xffffffffu, got, 0));
  }
  // Lane 0, after the walk.
  __device__ __forceinline__ void finish(const WaitCtx& ctx) {
    if (ok) publish(make_int4(-1, 0, 0, 0), ctx);
    if (more) item_drop_rest(q, answers, asked);
  }
};

// WARP: the reader is a whole converged warp, all of whose lanes leave together if a wait gives up; else one thread.
template <bool WARP>
struct ItemReader {
  ItemQueue* q;
  int n;   // entries read so far
  int4 e;  // the current one; its item is -1 after the last one (or after a wait that gave up)
  __device__ __forceinline__ ItemReader(ItemQueue& queue, const WaitCtx& ctx) : q(&queue), n(0) { next(ctx); }
  __device__ __forceinline__ int item() const { return e.x; }
  __device__ __forceinline__ void next(const WaitCtx& ctx) {
    const int s = n % kItemSlots;
    bool ok = mbar_wait(&q->full[s], (n / kItemSlots) & 1, ctx, kWaitItemFull);
    if (WARP) ok = __all_sync(0xffffffffu, ok);
    e = q->entry[s];
    if (!ok) e.x = -1;
    if (WARP) __syncwarp();
    if (!WARP || (threadIdx.x & 31) == 0) mbar_arrive(&q->empty[s]);
    ++n;
  }
};

// Four warps that read the same items and meet at named barriers.  A wait that gives up does so in one warp: another
// role has raised the abort flag, this warp's poll saw it, and a sibling's wait may still have succeeded.  A named barrier
// has no time limit, so the four leave together or not at all: before the barriers of an item they agree that each of them
// got there, and a warp that leaves its loop without that vote (no item for it: the end, or a wait that gave up) votes
// against.  Every warp's last vote is therefore a no of one of them, or, at the end, of all.
struct ReaderGroup {
  static constexpr int kThreads = 128;
  uint32_t barrier;
  bool apart;  // the group has voted no
  __device__ __forceinline__ explicit ReaderGroup(uint32_t named_barrier) : barrier(named_barrier), apart(false) {}
  // Once per item, before its first named barrier: whether all four go on.
  __device__ __forceinline__ bool agree(bool ok) {
    apart = !named_barrier_and(barrier, kThreads, ok);
    return !apart;
  }
  // After the loop over the items.
  __device__ __forceinline__ void leave() {
    if (!apart) named_barrier_and(barrier, kThreads, false);
  }
};

// Zeros into `rows` rows of BYTES bytes (at most 512), `stride` bytes apart, by a whole warp.
template <int BYTES>
__device__ __forceinline__ void warp_clear_rows(void* first, int64_t stride, int rows) {
  constexpr int kLanes = BYTES / 16;
  const int lane = threadIdx.x & 31;
  uint8_t* p = static_cast<uint8_t*>(first) + (lane / kLanes) * stride + (lane % kLanes) * 16;
#pragma unroll 4
  for (int i = lane / kLanes; i < rows; i += 32 / kLanes, p += (32 / kLanes) * stride) *reinterpret_cast<uint4*>(p) = make_uint4(0, 0, 0, 0);
}

}  // namespace sm100
}  // namespace kb
