// pair_tile.cuh -- how the FP64 density and force deal a particle's neighbour
// entries over a warp, and the ordered sums that follow.
//
// The reference sums each particle's neighbour terms in list order, farthest
// first, with a rounding per addition, so the additions of one particle are a
// chain; the terms themselves are independent and hold nearly all the work.
// A warp takes a tile of W particles and, chunk by chunk of their lists
// (farthest chunk first), computes the W x chunk terms with one lane per
// (particle, entry) pair, leaves them in shared memory, and then a lane per
// particle adds its terms in order.
//
// W follows the particle count: the warps the GPU holds at once take equal
// shares, of 32 particles at most. With few particles that is one or a few per
// warp: the terms of a particle's list run side by side in the lanes, where
// one thread per particle computed them one after the other in a few resident
// warps (N = 10,000: 313 warps on 608 sub-partitions).
#pragma once
#include <algorithm>

#include "physics.cuh"

namespace sphgpu {

constexpr int kPairSlots = 288;  // terms a warp's tile holds: W (chunk | 1) at most

// A row of ce terms is kept at an odd stride (in doubles), so that the lanes
// of the ordered sums, one row each, meet every bank pair once.
__host__ __device__ constexpr int pair_stride(int ce) { return ce | 1; }
// Entries per chunk at tile width W: the most, up to 32, whose rows fit.
__host__ __device__ constexpr int pair_chunk(int W, int slots) {
    const int t = slots / W, c = t & 1 ? t : t - 1;
    return c < 32 ? c : 32;
}
constexpr bool pair_rows_fit(int slots) {
    for (int W = 1; W <= 32; W++)
        for (int ce = 1; ce <= pair_chunk(W, slots); ce++)
            if (W * pair_stride(ce) > slots) return false;
    return true;
}

// The tiles of n particles on a GPU that holds `resident` warps at once: as
// many full passes of 32 particles a warp as there are, and the rest in equal
// shares, one per resident warp, or, up to `narrow` particles each, three per
// sub-partition: a tile's ordered sums are an addition instruction per entry of
// the list whatever its width, so that with one particle per warp the FP64 unit
// spends its time on them (density and force stage, us, one particle per
// resident warp and three warps per sub-partition: N = 2000 14.6, 18.4 and 12.5,
// 16.4; 4096 20.5, 20.5 and 14.4, 20.5; 10,000 22.0, 28.7 and 18.4, 28.7;
// density alone 24,000 30.7 and, at 10, 26.6). A tile is a block of one warp,
// so that the next tile starts as soon as a warp is free; with a resident
// block for every slot striding over the tiles, a pass of which a few warps had
// one tile more than the others left the rest idle.
struct PairTiles {
    int64_t full;  // tiles of 32 particles, first
    int W;         // width of the others
    int64_t n;
    PairTiles(int64_t n_, int sms, int warps_per_sm, int narrow) : n(n_) {
        const int64_t resident = (int64_t)sms * warps_per_sm, few = (int64_t)sms * 12;
        full = n / (32 * resident) * resident;
        const int64_t rest = n - 32 * full, share = (rest + resident - 1) / resident, wide = (rest + few - 1) / few;
        W = (int)std::max<int64_t>({share, std::min<int64_t>(wide, narrow), 1});
    }
    int grid() const { return (int)(full + (n - 32 * full + W - 1) / W); }
    // first particle of tile t, and its width
    __device__ __forceinline__ int64_t first(int64_t t, int &w) const {
        w = t < full ? 32 : W;
        return t < full ? 32 * t : 32 * full + (t - full) * W;
    }
};

// Chunk c = 0, 1, ... of a list of k entries, farthest first: entries
// [lo, lo + ce); the chunks' lengths differ by at most one.
struct PairChunks {
    int n, base, extra;  // chunks; shortest length; how many are one longer
    __device__ __forceinline__ PairChunks(int k, int W, int slots) {
        n = (k + pair_chunk(W, slots) - 1) / pair_chunk(W, slots);
        base = k / n;
        extra = k - base * n;
    }
    __device__ __forceinline__ int len(int c) const { return base + (c < extra ? 1 : 0); }
};

// i / ce for i < 1024, ce <= 32, given (65536 + ce - 1) / ce: exact, since the
// multiplier exceeds 65536 / ce by less than one and i < 65536 / ce.
__device__ __forceinline__ int pair_row(int i, int magic) { return (i * magic) >> 16; }

}  // namespace sphgpu
