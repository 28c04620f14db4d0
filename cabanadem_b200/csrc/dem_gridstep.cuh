// dem_gridstep.cuh -- the barrier that ends a step of a cooperative launch, with the step's largest
// |u|^2 and a count brought along (dem_live.cuh, dem_bonded.cu).
//
// Three rotating 16-byte words (scratch, zeroed before the launch): arrivals in the low half of the
// first 8 bytes and the count in the high half, the bits of the largest |u|^2 in the second 8.  A
// block folds its maximum, then arrives with a release; one atomic 16-byte acquire load polls both
// (bounded).  Block 0 clears the word of step k + 1 during step k: its last pollers (step k - 2)
// have arrived at the barrier of step k - 1.  Every block reads the same values, so decisions taken
// from them are the same.  About 1.2 us between blocks on a B200: two L2 round trips and the
// release's fence; the maximum read apart, after the poll, was another 400 cycles.  Per-block flags
// polled by a warp instead of one counter took 3.5 us at 118 blocks.
#pragma once
#include "dem_internal.cuh"

namespace b200dem {
namespace {

constexpr int kGridStepPolls = 1 << 22;

template <int BLOCK>
struct GridStep {   // in shared memory
    unsigned long long vmax[BLOCK / 32], arr, v2;
    int cnt[BLOCK / 32];
};

__device__ __forceinline__ void ld_acquire_b128(const void *p, unsigned long long &lo, unsigned long long &hi) {
    asm volatile(
        "{\n\t"
        ".reg .b128 t;\n\t"
        "ld.acquire.gpu.global.b128 t, [%2];\n\t"
        "mov.b128 {%0, %1}, t;\n\t"
        "}\n"
        : "=l"(lo), "=l"(hi)
        : "l"(p)
        : "memory");
}

// Largest of the warp's non-negative doubles, exactly: the high words, then the low words of those
// that share the largest high word.  A NaN counts as 0, as in finish_step (its bits would be the largest
// of all and end the displacement bound): the next list build reports it.
__device__ __forceinline__ unsigned long long warp_max_bits(double v) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    const unsigned long long b = (unsigned)(bits >> 32) > 0x7ff00000u ? 0ull : bits;   // past infinity: a NaN
    const unsigned hi = (unsigned)(b >> 32);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)b : 0u);
    return ((unsigned long long)mh << 32) | ml;
}

// Step k (0, 1, ... of the launch) ends: v2 >= 0 of the thread, count of the warp (the same in its
// lanes).  Returns false when the wait gave up (DEM_ERR_TIMEOUT is set); else `big` holds the bits of
// the grid's largest v2 and `total` the sum of the counts.  fc: the wait's limit, and whether blocks
// leave out their arrival, for testing it (dem_solver_debug_stream_waits).
template <int BLOCK>
__device__ __forceinline__ bool grid_step(GridStep<BLOCK> &s, Ctl *ctl, const ForceConsts &fc, unsigned long long *scratch,
                                          int k, double v2, int count, unsigned long long &big, int &total) {
    constexpr int W = BLOCK / 32;
    const unsigned long long one = fc.drop_copies ? 0ull : 1ull;
    const int limit = fc.wait_polls > 0 ? fc.wait_polls : kGridStepPolls;
    const unsigned long long vb = warp_max_bits(v2);
    if ((threadIdx.x & 31) == 0) {
        s.vmax[threadIdx.x >> 5] = vb;
        s.cnt[threadIdx.x >> 5] = count;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long *slot = scratch + 2 * (k % 3), vm = s.vmax[0];
        int c = s.cnt[0];
        for (int q = 1; q < W; ++q) {
            vm = s.vmax[q] > vm ? s.vmax[q] : vm;
            c += s.cnt[q];
        }
        if (blockIdx.x == 0) {
            unsigned long long *nxt = scratch + 2 * ((k + 1) % 3);
            nxt[0] = 0ull;
            nxt[1] = 0ull;
        }
        if (vm) atomicMax(&slot[1], vm);
        // the block's writes before its arrival
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(slot), "l"(one + ((unsigned long long)c << 32))
                     : "memory");
        unsigned long long arr, v;
        int p = 0;
        do ld_acquire_b128(slot, arr, v);
        while ((unsigned)arr < gridDim.x && ++p < limit);
        if (p == limit) {
            atomicOr(&ctl->status, DEM_ERR_TIMEOUT);
            arr = ~0ull;
        }
        s.arr = arr;
        s.v2 = v;
    }
    __syncthreads();   // every block has arrived (or this one gave up)
    const unsigned long long arr = s.arr;
    big = s.v2;
    total = (int)(arr >> 32);
    return arr != ~0ull;
}

}  // namespace
}  // namespace b200dem
