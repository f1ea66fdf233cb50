// grid_sync.cuh -- the grid-wide exchange of the cooperative kernels
// (k_coop in k_coop.cuh, k_adj_sweep in k_adjoint.cu).
//
// An exchange is a barrier over the grid that carries the maximum of one
// unsigned value per block.  Each block's thread 0 adds
// to one slot of memory {max, count} with reductions, the count last
// behind an acquire-release fence, and polls the slot (one 16-byte acquire
// load) until every block has counted.  Measured on 512-thread blocks that
// have just stored 2 KB each (cycles): 2400 with 32 blocks, 2730 with 152; a
// word per block that every block polls took 3600 and 4440 (a line per word;
// 7000 and 12,500 with the words in one line, which every store to it takes
// away from all pollers), a two-level tree 9600 and 11,200, clusters of eight
// with one polling CTA each 5400 (32 to 104 blocks).
//
// Four slots take turns, exchange X (counted over the life of the context, in 64
// bits: a small system makes 2^32 of them in hours)
// using slot X & 3; a slot's count grows by the grid size with every use, and
// its maximum is cleared for exchange X + 2 by block 0 after exchange X:
// every block that used them last (X - 2) has read them before it counted in
// X - 1, and none adds to them again before block 0 has counted in X + 1.
#pragma once
#include <cuda_runtime.h>

namespace femmd {

constexpr int kGridSlotWords = 16;  // 8-byte words from one slot to the next (a line each)
constexpr int kGridSlots = 4;
constexpr int kGridPolls = 1 << 20;  // polls (about 0.4 us each) before an exchange gives up

__device__ __forceinline__ unsigned long long *grid_slot(unsigned long long *base, unsigned long long x) {
    return base + (size_t)(x & (kGridSlots - 1)) * kGridSlotWords;
}

// Thread 0 of a block, after a block barrier that follows the block's stores:
// exchange x with 'blocks' blocks.  False when the wait gave up.  withhold:
// this block does not count (a test of the bounded wait).  After a block
// barrier that follows it, every store made by any block before its call is
// visible to the whole block.
__device__ __forceinline__ bool grid_exchange(unsigned long long *base, unsigned long long x, int blocks,
                                              unsigned value, bool withhold, unsigned &maxv) {
    unsigned long long *slot = grid_slot(base, x);
    if (value) asm volatile("red.relaxed.gpu.global.max.u32 [%0], %1;" ::"l"(slot), "r"(value) : "memory");
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    if (!withhold) asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(slot + 1), "l"(1ull) : "memory");
    const unsigned long long want = (x / kGridSlots + 1ull) * (unsigned long long)blocks;
    unsigned long long lo = 0ull, hi = 0ull;
    int it = 0;
    do {
        asm volatile("{\n .reg .b128 t;\n ld.acquire.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
                     : "=l"(lo), "=l"(hi)
                     : "l"(slot)
                     : "memory");
    } while (hi < want && ++it < kGridPolls);
    maxv = (unsigned)lo;
    if (blockIdx.x == 0) *reinterpret_cast<volatile unsigned long long *>(grid_slot(base, x + 2)) = 0ull;
    return hi >= want;
}

}  // namespace femmd
