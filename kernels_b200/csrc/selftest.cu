// kb_selftest_wait_timeout: runs the kernels' bounded device-side wait to its limit, on purpose and
// harmlessly, so that the give-up path (status words, abort flag, clean return) can be tested on a GPU.
//
// Every wait of the tcgen05 kernels is sm100::mbar_wait, which polls an mbarrier a bounded number of
// times, then records {KB_ERR_DEVICE_TIMEOUT, wait site, block} in the caller's status words, raises the
// CTA's abort flag and returns false; the roles then leave their loops and the kernel ends normally.  In
// a correct pipeline that path never runs.  This kernel makes it run in the smallest possible setting:
// one CTA whose only mbarrier expects an arrival that nobody makes, no copy in flight, no TMEM held, and
// a limit of 1 024 polls (well under a millisecond) instead of the kernels' 2^22.  Nothing faults and
// nothing hangs: the wait runs out, the second warp sees the abort flag the first one raised, the kernel
// returns and the context stays usable.
//
// kb_selftest_reader_group: the case in which only some of the warps that meet at named barriers see a wait give up.
// Two of four reader warps wait for an item that has not been published when the abort flag goes up; the other two look
// only after the first two have left, and find the item there.  All four must end their loops (ReaderGroup), so the
// kernel returns.  Every spin in it is bounded.
#include "common.cuh"
#include "item_queue.cuh"
#include "sm100_ptx.cuh"

namespace kb {
namespace {

using namespace sm100;

constexpr int kSelftestWaitSite = 900;
constexpr uint32_t kSelftestLimit = 1024;

__global__ void __launch_bounds__(64) wait_timeout_selftest_kernel(int32_t* status, int32_t* seen) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();
  const WaitCtx ctx{&abort_flag, status};
  if (threadIdx.x == 0) {
    // phase 0 of a barrier nobody arrives on: gives up after kSelftestLimit polls
    const bool ok = mbar_wait<0, kSelftestLimit>(&bar, 0, ctx, kSelftestWaitSite);
    seen[0] = ok ? 1 : 0;
  }
  if (threadIdx.x == 32) {
    // a second role waiting on the same barrier with the kernels' own (long) limit: it must leave as soon as
    // the first role has raised the abort flag, not after its own 2^22 polls
    const bool ok = mbar_wait(&bar, 0, ctx, kSelftestWaitSite + 1);
    seen[1] = ok ? 1 : 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) seen[2] = abort_flag;
}

// Warps 0-3 read, thread 128 writes.  seen[w]: the number of items warp w worked on; seen[4 + w]: the last item it found.
__global__ void __launch_bounds__(160) reader_group_selftest_kernel(int32_t* status, int32_t* seen) {
  __shared__ ItemQueue queue;
  __shared__ int abort_flag, gone;
  if (threadIdx.x == 0) {
    item_queue_init(queue, 4);
    abort_flag = gone = 0;
    fence_mbar_init();
  }
  __syncthreads();
  const WaitCtx ctx{&abort_flag, status};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto wait_for = [&](volatile int* word, int value) {  // (at most a few milliseconds)
    for (int spins = 0; *word < value && spins < 10000; ++spins) __nanosleep(200);
  };
  if (warp == 4) {
    if (lane == 0) {
      const PackedGrid unused{};
      ItemWriter<false> items(queue, unused, 1);  // (a fixed walk: nothing is asked of the hardware)
      items.publish(make_int4(5, 0, 0, 0), ctx);
      wait_for(&gone, 4);  // every warp has worked on item 5
      *ctx.abort_flag = 1;
      wait_for(&gone, 6);  // warps 0 and 1 have given up the wait for the next one
      items.publish(make_int4(7, 0, 0, 0), ctx);
      atomicAdd(&gone, 1);
    }
  } else {
    ReaderGroup group(1);
    int done = 0, found = -1;
    bool ok = true;
    for (ItemReader<true> items(queue, ctx); ok && items.item() >= 0; items.next(ctx)) {
      found = items.item();
      ok = group.agree(true);
      if (!ok) break;
      ++done;
      named_barrier_sync(1, 128);
      if (lane == 0) atomicAdd(&gone, 1);
      if (warp >= 2) wait_for(&gone, 7);
    }
    if (warp < 2 && lane == 0) atomicAdd(&gone, 1);
    group.leave();
    if (lane == 0) {
      seen[warp] = done;
      seen[4 + warp] = found;
    }
  }
  __syncthreads();
}

}  // namespace
}  // namespace kb

extern "C" int kb_selftest_wait_timeout(int32_t* status, int32_t* seen, void* stream) {
  if (!status || !seen) return KB_ERR_BAD_ARGUMENT;
  kb::wait_timeout_selftest_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(status, seen);
  KB_LAUNCH_CHECK("wait_timeout_selftest_kernel");
  return KB_OK;
}

extern "C" int kb_selftest_reader_group(int32_t* status, int32_t* seen, void* stream) {
  if (!status || !seen) return KB_ERR_BAD_ARGUMENT;
  kb::reader_group_selftest_kernel<<<1, 160, 0, static_cast<cudaStream_t>(stream)>>>(status, seen);
  KB_LAUNCH_CHECK("reader_group_selftest_kernel");
  return KB_OK;
}
