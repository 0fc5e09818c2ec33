// k_bin.cu -- cell binning: the GB300 replacement of the reference's spatial
// index (sim/core.go:126-224 Partition/Treebuild, rebuilt on every force
// evaluation at sim/sph.go:406). Instead of a pointer tree it builds, per
// simulation, a dense Morton-ordered cell table at a fine level: drift +
// cell key + histogram (one atomic per particle, whose return value is the
// particle's rank inside its cell), an exclusive scan of the histogram into
// cell starts, and a permute of the state into cell order. Every coarser
// level's cell is a contiguous range of the same table, which is what the
// neighbour search walks. With many particles the passes are HBM streams; with
// few, each is a launch of about 2 us, so they are few: keys, scan (with the
// grouping by cell while one block can do both), permute.
#include "common.cuh"

#include <algorithm>

namespace sphgpu {

// Blocks for a pass over n particles: small ones for few particles, so that
// they spread over the SMs.
struct Pass {
    int grid, block;
    Pass(const Launch &L, int64_t n) : block(n <= 32768 ? 64 : 256) {
        grid = (int)std::min<int64_t>((n + block - 1) / block, (int64_t)L.sms * 8);
    }
};

// ------------------------------------------------------------------ bbox
// Bounding box of the predicted positions, for simulations with an open axis,
// as ordered 64-bit keys. A block takes one contiguous range of slots, so
// nearly every block (and nearly every warp of the others) lies in a single
// simulation; its threads reduce their keys first and one of them does the
// four atomics. With four atomics per particle, all on the same words, the
// kernel took 760 us at N = 300,000 (170 at 65,537).
__device__ __forceinline__ unsigned long long key_min(unsigned long long a, unsigned long long b) { return a < b ? a : b; }
__device__ __forceinline__ unsigned long long key_max(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

struct BoxKeys {
    unsigned long long k[4];  // min x, max x, min y, max y
    __device__ __forceinline__ void clear() { k[0] = k[2] = ~0ull; k[1] = k[3] = 0ull; }
    __device__ __forceinline__ void add(double2 p) {
        const unsigned long long x = dkey(p.x), y = dkey(p.y);
        k[0] = key_min(k[0], x);
        k[1] = key_max(k[1], x);
        k[2] = key_min(k[2], y);
        k[3] = key_max(k[3], y);
    }
    __device__ __forceinline__ void reduce_warp() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const unsigned long long v = __shfl_xor_sync(0xffffffffu, k[i], o);
                k[i] = i & 1 ? key_max(k[i], v) : key_min(k[i], v);
            }
        }
    }
    __device__ __forceinline__ void flush(const SimDev &S, SimDev &W) const {
        if (!S.periodic[0]) { atomicMin(&W.bbox[0], k[0]); atomicMax(&W.bbox[1], k[1]); }
        if (!S.periodic[1]) { atomicMin(&W.bbox[2], k[2]); atomicMax(&W.bbox[3], k[3]); }
    }
};

// Grid of open axes from the bounding box, and the FP32 fields that follow from
// it (as simdev_floats sets them). One thread's chain: an FP64 instruction takes
// 75 cycles for one lane as for 32, so products, quotients and conversions run
// on the integer pipes and nothing is computed that the box does not change
// (a hundred FP64 instructions before; step at N = 1000 44.2 -> 42.6 us).
__device__ void grid_one(SimDev &S, const BoxKeys &b) {
    const int G = 1 << S.level;
    double mag = 0.0, Lm = 0.0;
    auto size = [](double a) { return emu_double(emu_bits(a) & ~kEmuSign); };
    auto above = [](double a, double b) { return emu_bits(a) > emu_bits(b); };  // of numbers not negative
    for (int ax = 0; ax < 2; ax++) {
        if (!S.periodic[ax]) {
            double mn = dkey_inv(b.k[2 * ax]), mx = dkey_inv(b.k[2 * ax + 1]);
            if (!(mn <= mx)) { mn = 0; mx = 1; }
            double w = mx - mn;
            if (!(w > 0)) w = 1e-300 + fabs(mn) * 1e-12 + 1e-12;
            const double L = __fma_rn(w, 1.0 + 1e-9, 1e-300);
            S.lo[ax] = mn;
            S.L[ax] = L;
            S.s[ax] = emu_mul(L, emu_double((uint64_t)(1023 - S.level) << 52));
            S.inv_s[ax] = emu_div((double)G, emu_divisor(L), L);
            S.fs[ax] = emu_d2f(S.s[ax]);
            S.fdtc[ax] = emu_d2f(emu_mul(S.dth, S.inv_s[ax]));
        }
        const double L = S.L[ax], lo = size(S.lo[ax]), hi = size(__dadd_rn(S.lo[ax], L));
        double m = __dadd_rn(above(lo, hi) ? lo : hi, L);
        if (!emu_is_zero(S.dimg[ax])) m = __dadd_rn(m, size(S.dimg[ax]));
        if (above(m, mag)) mag = m;
        if (above(L, Lm)) Lm = L;
    }
    S.flmax = emu_d2f(Lm);
    S.fmag = emu_d2f(mag);
    S.tol = emu_d2f(emu_mul(Lm, 4.0e-7));
}

// The last block to finish turns the boxes into grids; it takes the ticket back
// to zero for the next launch.
__device__ __forceinline__ void last_block_grids(const Ctx &c) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(c.flags + 1, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int s = threadIdx.x; s < c.nsims; s += blockDim.x) {
        SimDev &S = c.sims_rw[s];
        grid_one(S, BoxKeys{{__ldcg(&S.bbox[0]), __ldcg(&S.bbox[1]), __ldcg(&S.bbox[2]), __ldcg(&S.bbox[3])}});
    }
    if (threadIdx.x == 0) c.flags[1] = 0u;
}

__global__ void __launch_bounds__(256) k_bbox(Ctx c, PArrays A, int pred) {
    __shared__ BoxKeys part[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t per = (c.n + gridDim.x - 1) / gridDim.x;
    const int64_t i0 = min(c.n, blockIdx.x * per), i1 = min(c.n, i0 + per);
    const int s0 = sim_of(c, min(i0, c.n - 1));
    const bool one = i0 >= i1 || s0 == sim_of(c, i1 - 1);  // slots are ordered by simulation
    BoxKeys b;
    b.clear();
    for (int64_t base = i0; base < i1; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        if (!one) b.clear();
        int s = s0;
        if (i < i1) {
            s = sim_of(c, i);
            double2 p = A.pos[i];
            if (pred == PRED_DRIFT) {  // predict()'s position
                const double2 v = A.vel[i];
                const double dth = c.sims[s].dth;
                p.x = __dadd_rn(p.x, emu_mul(v.x, dth));
                p.y = __dadd_rn(p.y, emu_mul(v.y, dth));
            }
            b.add(p);
        }
        if (!one) {
            const uint32_t live = __ballot_sync(0xffffffffu, i < i1);
            const int first = __shfl_sync(0xffffffffu, s, 0);
            if (__all_sync(0xffffffffu, i >= i1 || s == first)) {
                b.reduce_warp();
                if (live && lane == 0) b.flush(c.sims[first], c.sims_rw[first]);
            } else if (i < i1) {
                b.flush(c.sims[s], c.sims_rw[s]);
            }
        }
    }
    if (one) {
        b.reduce_warp();
        if (lane == 0) part[w] = b;
        __syncthreads();
        if (w == 0) {
            if (lane < (int)(blockDim.x >> 5)) b = part[lane];
            else b.clear();
            b.reduce_warp();
            if (lane == 0) b.flush(c.sims[s0], c.sims_rw[s0]);
        }
    }
    last_block_grids(c);
}

void launch_bbox(const Ctx &c, const Launch &L, const PArrays &A, int pred) {
    k_bbox<<<(int)std::min<int64_t>((c.n + 255) / 256, (int64_t)L.sms * 4), 256, 0, L.stream>>>(c, A, pred);
}

// ------------------------------------------------------------------- bin
__global__ void k_bin(Ctx c, PArrays A, Tables T, int32_t *ndefer, int pred) {
    // the search's counts start over (sph_search_stats reads them until then);
    // a memset node between the kernels of the graph cost 4 to 6 us a step
    // (mixed N = 10,000 57 -> 53 us, tank 65,537 158 -> 152)
    if (ndefer && blockIdx.x == 0 && threadIdx.x < 2) ndefer[threadIdx.x] = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < c.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        int s = sim_of(c, i);
        const SimDev &S = c.sims[s];
        // The cell of the drifted position, in cell units: the offset from the
        // grid origin in FP64, rounded once to FP32 (error <= 2^-24 G cells,
        // 6e-8 L), plus the drift vel * dth in FP32. The exact FP64 drift is
        // k_permute's; a particle within that error of a cell face may land in
        // the neighbouring cell, which the searches' slack S.tol (4e-7 L)
        // covers. The FP64 unit would be the binning's bound (each instruction, a
        // conversion included, holds it for 75 cycles of a sub-partition): the
        // conversions run on the integer pipes, and where the grid starts at 0
        // and its cells per unit are a power of two (a unit box), the offset's
        // subtraction and scaling are exact and need no FP64 at all. (Binning
        // pass, N = 1,048,576 24 -> 17 us, 4,194,304 81 -> 60.)
        const double2 pos = A.pos[i];
        float tx = S.fcell[0] != 0.f ? emu_d2f(pos.x) * S.fcell[0] : emu_d2f(__dmul_rn(__dsub_rn(pos.x, S.lo[0]), S.inv_s[0]));
        float ty = S.fcell[1] != 0.f ? emu_d2f(pos.y) * S.fcell[1] : emu_d2f(__dmul_rn(__dsub_rn(pos.y, S.lo[1]), S.inv_s[1]));
        if (pred == PRED_DRIFT) {
            const double2 vel = A.vel[i];
            tx = __fmaf_rn(emu_d2f(vel.x), S.fdtc[0], tx);
            ty = __fmaf_rn(emu_d2f(vel.y), S.fdtc[1], ty);
        }
        if (!isfinite(tx) || !isfinite(ty)) atomicOr(c.flags, (unsigned)FLAG_NONFINITE);
        const int G = 1 << S.level;
        const float Gf = (float)G;
        const int cx = !(tx >= 0.f) ? 0 : tx >= Gf ? G - 1 : (int)tx;
        const int cy = !(ty >= 0.f) ? 0 : ty >= Gf ? G - 1 : (int)ty;
        // distance outside the periodic domain (the wrap moves at most one axis per step)
        float o = 0.f;
        if (S.periodic[0]) o = fmaxf(o, fmaxf(-tx, tx - Gf) * S.fs[0]);
        if (S.periodic[1]) o = fmaxf(o, fmaxf(-ty, ty - Gf) * S.fs[1]);
        if (o > 0.f) atomicMax((int *)&c.sims_rw[s].overshoot, __float_as_int(o * 1.0001f));
        int32_t key = (int32_t)(S.cell_off + morton2(cx, cy));
        T.key[i] = key;
        T.rank[i] = atomicAdd(&T.count[key], 1);
    }
}

void launch_bin(const Ctx &c, const Launch &L, const PArrays &A, const Tables &T, int32_t *ndefer, int pred) {
    const Pass p(L, c.n);
    k_bin<<<p.grid, p.block, 0, L.stream>>>(c, A, T, ndefer, pred);
}

// ---------------------------------------------------------- stable order
// The histogram's atomic ranks order a cell's particles arbitrarily. To make
// every later order (and so every floating-point sum) reproducible, each
// particle's slot inside its cell is its rank by index in the previous order
// among the cell's members: the members are grouped by cell (which also zeroes
// the touched counts for the next binning), then every particle counts the
// members of its cell with a smaller index (in the permute). Both are per
// particle, so their cost does not grow with the cell table (the k = 64 stress
// workload bins into 4^14 mostly empty cells).
__device__ __forceinline__ void group_one(const Tables &T, int64_t i) {
    const int32_t key = T.key[i];
    T.tmp[T.start[key] + T.rank[i]] = (int32_t)i;
    T.count[key] = 0;
}

__global__ void k_group(Ctx c, Tables T) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < c.n;
         i += (int64_t)gridDim.x * blockDim.x)
        group_one(T, i);
}

// ------------------------------------------------------------------ scan
// Exclusive scan of the cell counts into cell starts, over tiles of kScanTile
// cells: one block for small tables; tile sums and then starts while a block
// can add up the sums before its own (a few KB from L2); with a pass over the
// sums between for the largest. The counts are zeroed per particle afterwards
// (grouping), so the passes over the whole cell table only read counts and
// write starts.
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int64_t kScanOneBlockCells = 16384;  // (scan stage at 65,536 cells: 38 us against 12)
constexpr int kScanDirectTiles = 4096;
constexpr int64_t kGroupOneBlockN = 4096;  // (16,000 particles: step 97 us against 94 with a launch of its own)
constexpr int64_t kRankPassN = 524288;  // beyond, the ranks are a pass of their own (step at 200,001: 707 us with, 704 without)

__device__ __forceinline__ int block_exclusive_scan(int v, int *warp_sums, int &total) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        int nw = blockDim.x >> 5;
        int t = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) warp_sums[lane] = t;
    }
    __syncthreads();
    total = warp_sums[(blockDim.x >> 5) - 1];
    int before = w > 0 ? warp_sums[w - 1] : 0;
    int r = before + x - v;
    __syncthreads();
    return r;
}

// A thread's eight consecutive cells (32-byte aligned) as two 16-byte loads;
// cells past the end read as empty.
__device__ __forceinline__ void load_counts(const Tables &T, int64_t base, int (&v)[kScanItems]) {
    if (base + kScanItems <= T.ncells) {
        const int4 a = *reinterpret_cast<const int4 *>(T.count + base);
        const int4 b = *reinterpret_cast<const int4 *>(T.count + base + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < kScanItems; j++) v[j] = base + j < T.ncells ? T.count[base + j] : 0;
    }
}

__global__ void k_scan_tiles(Tables T) {
    __shared__ int ws[32];
    int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int v[kScanItems];
    load_counts(T, base, v);
    int sum = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) sum += v[j];
    int total;
    block_exclusive_scan(sum, ws, total);
    if (threadIdx.x == 0) T.partial[blockIdx.x] = total;
}

__global__ void k_scan_partials(Tables T, int ntiles) {
    __shared__ int ws[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b = 0; b < ntiles; b += blockDim.x) {
        int idx = b + threadIdx.x;
        int v = idx < ntiles ? T.partial[idx] : 0;
        int total;
        int ex = block_exclusive_scan(v, ws, total);
        if (idx < ntiles) T.partial[idx] = ex + carry;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) T.start[T.ncells] = carry;
}

// DIRECT: partial holds the tiles' own sums; else their exclusive scan
template <bool DIRECT>
__global__ void k_scan_final(Tables T) {
    __shared__ int ws[32];
    int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int v[kScanItems];
    load_counts(T, base, v);
    int before = 0;
    if (DIRECT) {
        int mine = 0;
        for (int b = threadIdx.x; b < (int)blockIdx.x; b += kScanThreads) mine += T.partial[b];
        block_exclusive_scan(mine, ws, before);
    } else {
        before = T.partial[blockIdx.x];
    }
    int sum = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) sum += v[j];
    int total;
    int ex = block_exclusive_scan(sum, ws, total) + before;
    if (DIRECT && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) T.start[T.ncells] = before + total;
    int st[kScanItems];
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        st[j] = ex;
        ex += v[j];
    }
    if (base + kScanItems <= T.ncells) {
        *reinterpret_cast<int4 *>(T.start + base) = make_int4(st[0], st[1], st[2], st[3]);
        *reinterpret_cast<int4 *>(T.start + base + 4) = make_int4(st[4], st[5], st[6], st[7]);
    } else {
#pragma unroll
        for (int j = 0; j < kScanItems; j++)
            if (base + j < T.ncells) T.start[base + j] = st[j];
    }
}

// A table of at most kScanOneBlockCells cells by one block, and with it (group)
// the particles' grouping by cell.
__global__ void __launch_bounds__(1024) k_scan_one(Ctx c, Tables T, int group) {
    __shared__ int ws[32];
    const int nc = (int)T.ncells, per = ((nc + 1023) / 1024 + 3) & ~3;  // whole 16-byte words of counts
    const int x0 = min((int)threadIdx.x * per, nc), x1 = min(x0 + per, nc);
    int sum = 0;
    if ((nc & 3) == 0) {
        for (int x = x0; x < x1; x += 4) {
            const int4 v = *reinterpret_cast<const int4 *>(T.count + x);
            sum += v.x + v.y + v.z + v.w;
        }
    } else {
        for (int x = x0; x < x1; x++) sum += T.count[x];
    }
    int total;
    int run = block_exclusive_scan(sum, ws, total);
    if (threadIdx.x == 0) T.start[nc] = total;
    if ((nc & 3) == 0) {
        for (int x = x0; x < x1; x += 4) {
            const int4 v = *reinterpret_cast<const int4 *>(T.count + x);
            *reinterpret_cast<int4 *>(T.start + x) = make_int4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
            run += v.x + v.y + v.z + v.w;
        }
    } else {
        for (int x = x0; x < x1; x++) {
            T.start[x] = run;
            run += T.count[x];
        }
    }
    if (!group) return;
    __syncthreads();
    for (int i = threadIdx.x; i < (int)c.n; i += 1024) group_one(T, i);
}

// A particle's slot: the cell's first plus the members with a smaller index.
__device__ __forceinline__ int slot_of(const Tables &T, int64_t i) {
    const int32_t key = T.key[i];
    const int x0 = T.start[key], x1 = T.start[key + 1];
    int d = x0;
    for (int x = x0; x < x1; x++) d += T.tmp[x] < (int32_t)i ? 1 : 0;
    return d;
}

__global__ void k_rank(Ctx c, Tables T) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < c.n;
         i += (int64_t)gridDim.x * blockDim.x)
        T.rank[i] = slot_of(T, i);
}

// starts, the particles grouped by cell, and (many particles) their slots
void launch_scan(const Ctx &c, const Launch &L, const Tables &T) {
    const bool one = T.ncells <= kScanOneBlockCells, group = one && c.n <= kGroupOneBlockN;
    if (one) {
        k_scan_one<<<1, 1024, 0, L.stream>>>(c, T, group ? 1 : 0);
    } else {
        const int ntiles = (int)((T.ncells + kScanTile - 1) / kScanTile);
        k_scan_tiles<<<ntiles, kScanThreads, 0, L.stream>>>(T);
        if (ntiles <= kScanDirectTiles) {
            k_scan_final<true><<<ntiles, kScanThreads, 0, L.stream>>>(T);
        } else {
            k_scan_partials<<<1, 1024, 0, L.stream>>>(T, ntiles);
            k_scan_final<false><<<ntiles, kScanThreads, 0, L.stream>>>(T);
        }
    }
    const Pass p(L, c.n);
    if (!group) k_group<<<p.grid, p.block, 0, L.stream>>>(c, T);
    if (c.n > kRankPassN) k_rank<<<p.grid, p.block, 0, L.stream>>>(c, T);
}

// --------------------------------------------------------------- permute
// Writes the predicted state into cell order (B), plus the float-pair
// position record relative to the grid origin used by the FP32 distance
// filter and the mixed-precision sums, and (velrec) the predicted
// velocity as float pairs.
template <bool RANKED>
__global__ void k_permute(Ctx c, PArrays A, PArrays B, Tables T, int pred, int velrec) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < c.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        int s = sim_of(c, i);
        const SimDev &S = c.sims[s];
        const int64_t d = RANKED ? T.rank[i] : slot_of(T, i);
        double2 pos = A.pos[i], vel = A.vel[i];
        double u = A.u[i];
        double2 p, vp;
        double up;
        predict(S, pred, pos, vel, A.acc[i], u, A.udot[i], A.vp[i], A.up[i], p, vp, up);
        B.pos[d] = p;
        B.vel[d] = vel;
        B.vp[d] = vp;
        B.u[d] = u;
        B.up[d] = up;
        B.id[d] = A.id[i];
        B.hprev[d] = A.hprev[i];
        float4 r;
        split_df(__dsub_rn(p.x, S.lo[0]), r.x, r.z);
        split_df(__dsub_rn(p.y, S.lo[1]), r.y, r.w);
        B.rec[d] = r;
        if (velrec) {
            float4 v;
            split_df(vp.x, v.x, v.z);
            split_df(vp.y, v.y, v.w);
            B.vrec[d] = v;
        }
    }
}

void launch_permute(const Ctx &c, const Launch &L, const PArrays &A, const PArrays &B,
                    const Tables &T, int pred, bool velrec) {
    // a block per 256 particles: the copies of this pass, unlike the binning's
    // atomics and scattered ids, gain from blocks in order (clustered
    // N = 4,194,304 130 -> 121 us against 8 striding blocks per SM; the binning
    // pass then takes 67 instead of 60)
    const int block = Pass(L, c.n).block, grid = (int)((c.n + block - 1) / block);
    // the ranks' loads in front of the drift cost more than a launch once the
    // arrays outgrow L2 (clustered N = 4,194,304: 165 us against 130 + 21)
    if (c.n > kRankPassN) k_permute<true><<<grid, block, 0, L.stream>>>(c, A, B, T, pred, velrec ? 1 : 0);
    else k_permute<false><<<grid, block, 0, L.stream>>>(c, A, B, T, pred, velrec ? 1 : 0);
}

}  // namespace sphgpu
