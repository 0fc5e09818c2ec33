// pair_tile.cuh -- how the FP64 density and force deal a particle's neighbour
// entries over a warp, and the ordered sums that follow.
//
// The reference sums each particle's neighbour terms in list order, farthest
// first, with a rounding per addition, so the additions of one particle are a
// chain; the terms themselves are independent and hold nearly all the work.
// A warp takes a tile of W particles and, chunk by chunk of at most 32 / W * 8
// entries (farthest chunk first), computes the W x chunk terms with one lane
// per (particle, entry) pair, leaves them in shared memory, and then a lane per
// particle adds its terms in order.
//
// W = 32 when there are enough particles to fill the GPU (the ordered sums
// then use all lanes, as one thread per particle would); fewer particles take
// a smaller W, down to one particle per warp: the terms of a particle's list
// run side by side in the lanes, where one thread per particle computed them
// one after the other in a few resident warps (N = 10,000: 313 warps on 608
// sub-partitions).
#pragma once
#include "physics.cuh"

namespace sphgpu {

constexpr int kPairWarps = 4;    // warps per block (each works alone)
constexpr int kPairSlots = 288;  // terms a warp's tile holds: W (chunk | 1) at most

// Entries per chunk at tile width W.
__host__ __device__ constexpr int pair_chunk(int W) { return W >= 32 ? 8 : W >= 16 ? 16 : 32; }
// A row of ce terms is kept at an odd stride (in doubles), so that the lanes
// of the ordered sums, one row each, meet every bank pair once.
__host__ __device__ constexpr int pair_stride(int ce) { return ce | 1; }
static_assert(32 * pair_stride(8) <= kPairSlots && 16 * pair_stride(16) <= kPairSlots && 8 * pair_stride(32) <= kPairSlots,
              "a tile's terms fit its slots at every width");

// The smallest power of two that covers n particles with the warps the GPU
// holds at once, at most 32.
inline int pair_width(int64_t n, int64_t resident_warps) {
    int W = 1;
    while (W < 32 && (int64_t)W * resident_warps < n) W *= 2;
    return W;
}

// Chunk c = 0, 1, ... of a list of k entries, farthest first: entries
// [lo, lo + ce); the chunks' lengths differ by at most one.
struct PairChunks {
    int n, base, extra;  // chunks; shortest length; how many are one longer
    __device__ __forceinline__ PairChunks(int k, int W) {
        n = (k + pair_chunk(W) - 1) / pair_chunk(W);
        base = k / n;
        extra = k - base * n;
    }
    __device__ __forceinline__ int len(int c) const { return base + (c < extra ? 1 : 0); }
};

// i / ce for i < 1024, ce <= 32, given (65536 + ce - 1) / ce: exact, since the
// multiplier exceeds 65536 / ce by less than one and i < 65536 / ce.
__device__ __forceinline__ int pair_row(int i, int magic) { return (i * magic) >> 16; }

}  // namespace sphgpu
