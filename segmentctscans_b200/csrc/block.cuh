// What the threads of a block agree on.  tests/cpp/block_check.cpp compiles this file for the host and
// runs it with threads that advance in unfavourable orders.
#pragma once

#include <cstdint>

namespace potts {

constexpr int kPlainThreads = 256;

// A barrier of the block, and whether a wait of any thread had given up before it: the same answer in
// every thread.  (Read behind the barrier, the flag may already be set by a warp that has gone on to its
// next wait, and the warps leave their loop at different barriers.)
__device__ __forceinline__ bool sync_aborted(const volatile int *abort) { return __syncthreads_or(*abort) != 0; }

// The voxels of a block that need the projection loop: N floats each and the offset, column by
// column (threads of a warp write and read different banks).  A block walks kLoopChunks chunks of
// kPlainThreads voxels and runs the list when the next chunk might not fit (kCap entries, in 40 KB)
// and at its end.
constexpr int kLoopChunks = 4;
template <int N>
struct LoopList {
    static constexpr int kCap = (N + 2) * 4 * 512 <= 40 * 1024 ? 512 : 256;
    int64_t off[kCap];
    float v[N][kCap];
    int count;  // entries handed out since the list was last emptied

    // The entry of this thread's voxel (need: it has one); every thread of a warp calls it.
    __device__ __forceinline__ int add(bool need)
    {
        const unsigned m = __ballot_sync(0xffffffffu, need);
        const int lane = threadIdx.x & 31;
        int first = 0;
        if (lane == 0 && m) first = atomicAdd(&count, __popc(m));
        return __shfl_sync(0xffffffffu, first, 0) + __popc(m & ((1u << lane) - 1u));
    }
    // run(i) for every entry when the list is to be emptied; every thread of the block calls it after
    // each chunk, with its own `need` of the chunk and its own n, 0 at first: the entries in the list.
    // n comes from the barrier and not from `count`, which a warp that has left may raise for the next
    // chunk before the last warp reads it: all threads must empty the list, or none.
    template <typename Run>
    __device__ __forceinline__ void flush(int &n, bool need, bool last, Run run)
    {
        n += __syncthreads_count(need);
        if (!last && n <= kCap - kPlainThreads) return;
        if (threadIdx.x == 0) count = 0;  // the next add is behind the barrier below
        for (int i = (int)threadIdx.x; i < n; i += kPlainThreads) run(i);
        n = 0;
        __syncthreads();
    }
};

}  // namespace potts
