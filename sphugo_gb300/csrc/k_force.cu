// k_force.cu -- pressure + artificial-viscosity acceleration and du/dt
// (sim/sph.go:327-401 AccelerationAndEDot2D) fused with the rest of the
// leapfrog step (sim/sph.go:121-193: kick, drift, periodic wrap,
// reflections). The mixed form: one thread per particle walks its k
// neighbours from the farthest to the nearest. The FP64 form: the pairs dealt
// over the lanes, their terms added in that order.
#include "pair_tile.cuh"

#include <algorithm>

namespace sphgpu {

// Particles up to which the mixed force deals its pairs over the lanes (force
// stage with and without: N = 1000 12 and 18 us, 10,000 17 and 20, 20,000 20
// and 20, 100,000 39 and 29: a thread per particle then fills the GPU, and
// the factors' way through shared memory costs issue slots).
constexpr int64_t kMixedPairsMaxN = 16384;
constexpr int kMixedBlocks = 20;  // resident blocks (warps) per SM (8 KB each)
// The FP64 force is compiled twice: with 92 registers and chunks of nine entries
// at 32 particles, 20 warps resident per SM, and with 72 and seven, 25 resident.
// The second hides more latency, but each of its warps takes longer: it runs
// beyond one pass of its own (121,600 particles), except where the first takes
// just two (97,280 each; from one and a half of the second's on, up to 204,288):
// there the first took 0.95 to 1.00 of the second's time at k = 16, 32 and 45,
// 0.98 to 1.02 at 21, 0.98 to 1.04 at 64 (N = 183,000 to 204,000, uniform and
// clustered).
// Force stage, us, first and second: N = 50,000 81 and 86, 100,000 133 and 140,
// 110,000 137 and 157; 130,000 173 and 167, 140,000 185 and 171, 170,000 212
// and 205; 200,000 237 and 243; 250,000 303 and 290, 300,000 338 and 330,
// 500,000 544 and 533, 1,048,576 1103 and 1034, clustered 4,194,304 4262 and
// 4040; the same at k = 16, 45 and 64 (N = 110,000, 140,000, 200,000: k = 64 268
// and 315, 367 and 342, 464 and 481). 192 slots at 26 warps 1080 and 4112, 160
// at 30 (64 registers, spills) 1103 and 4203.
constexpr int kForceBlocks = 20, kForceBlocksMany = 25;
constexpr int kForceSlotsMany = 224;
// (force stage at N = 16,000: 35 us at six particles per warp, 37 at eight, 39 at ten)
constexpr int kForceNarrow = 6;
// Tiles up to this width sum with three lanes per particle: 29 us at N = 10,000
// against 40 with one.
constexpr int kSplitWidth = 10;

struct ForceArgs {
    Ctx c;
    PArrays B;  // positions / predictions of this evaluation (cell order)
    PArrays A;  // state written here (same order)
    Derived D;
    int integrate;
};

// x < y for x, y not NaN, on the integer pipes (an FP64 compare costs the FP64
// unit as much as an addition): the order of the bits read as integers, the
// negative ones mirrored (-0 onto 0).
__device__ __forceinline__ int64_t order_key(double x) {
    const int64_t b = (int64_t)emu_bits(x);
    return b < 0 ? (int64_t)(kEmuSign - (uint64_t)b) : b;
}
__device__ __forceinline__ bool less(double x, double y) { return order_key(x) < order_key(y); }
__device__ __forceinline__ bool is_nan(double x) { return (emu_bits(x) & ~kEmuSign) > 0x7ff0000000000000ull; }
__device__ __forceinline__ bool is_finite(double x) { return (emu_hi(x) & 0x7ff00000u) != 0x7ff00000u; }

// sim/sph.go:121-193 with two roundings per multiply-add: five additions on
// the FP64 unit, the products and compares on the integer pipes (the bounds
// are never NaN; a NaN position compares false)
__device__ __forceinline__ void integrate_one(const SimDev &S, double2 &pos, double2 &vel, double &u,
                                              double ax, double ay, double udot) {
    const double dth = S.dth;
    const double dt2 = emu_mul(2.0, dth);
    vel.x = __dadd_rn(vel.x, emu_mul(ax, dt2));
    vel.y = __dadd_rn(vel.y, emu_mul(ay, dt2));
    u = __dadd_rn(u, emu_mul(emu_mul(udot, 2.0), dth));
    pos.x = __dadd_rn(pos.x, emu_mul(vel.x, dth));
    pos.y = __dadd_rn(pos.y, emu_mul(vel.y, dth));
    const bool fx = !is_nan(pos.x), fy = !is_nan(pos.y);
    // periodic wrap: an if/continue chain, at most one axis per step
    if (fx && less(pos.x, S.per_lo[0])) pos.x = __dadd_rn(pos.x, __dsub_rn(S.per_hi[0], S.per_lo[0]));
    else if (fx && less(S.per_hi[0], pos.x)) pos.x = __dsub_rn(pos.x, __dsub_rn(S.per_hi[0], S.per_lo[0]));
    else if (fy && less(pos.y, S.per_lo[1])) pos.y = __dadd_rn(pos.y, __dsub_rn(S.per_hi[1], S.per_lo[1]));
    else if (fy && less(S.per_hi[1], pos.y)) pos.y = __dsub_rn(pos.y, __dsub_rn(S.per_hi[1], S.per_lo[1]));
    // reflections: Pos -= Pos - bound; Vel = -Vel
    if (fx && less(pos.x, S.refl[0])) { pos.x = __dsub_rn(pos.x, __dsub_rn(pos.x, S.refl[0])); vel.x = emu_neg(vel.x); }
    if (fx && less(S.refl[1], pos.x)) { pos.x = __dsub_rn(pos.x, __dsub_rn(pos.x, S.refl[1])); vel.x = emu_neg(vel.x); }
    if (fy && less(pos.y, S.refl[2])) { pos.y = __dsub_rn(pos.y, __dsub_rn(pos.y, S.refl[2])); vel.y = emu_neg(vel.y); }
    if (fy && less(S.refl[3], pos.y)) { pos.y = __dsub_rn(pos.y, __dsub_rn(pos.y, S.refl[3])); vel.y = emu_neg(vel.y); }
}

// The mixed form, one thread per particle. Bound by its neighbour gathers (ncu,
// uniform blast N = 1,048,576: L1 data path 69 % busy, 9 cycles of waiting on
// loads per issued instruction); 80 registers: at the 10 or 12 resident blocks
// that fewer would allow it ran 271 and 328 us against 217. A block per 128
// particles, not 16 blocks per SM striding over them: 217 -> 204, clustered
// N = 4,194,304 790 -> 730; records loaded one or two pairs ahead: 260 to 335.
__global__ void __launch_bounds__(128, 6) k_force_mixed(ForceArgs a) {
    const int k = a.c.k;
    const PArrays &B = a.B;
    const Derived &D = a.D;
    unsigned fl = 0;
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q < a.c.n) {
        const int s = sim_of(a.c, q);
        const SimDev &S = a.c.sims[s];
        const double2 P = B.pos[q];
        const int32_t *nb = D.nbr + q * k;
        double axo, ayo, edot;
        {
            // FP32 throughout the sums and prefactors (no FP64 work per particle
            // before the integrator)
            const float4 di = D.derf[q];
            const float ci = di.x, rhoi = di.y, hif = di.z, caf = di.w;
            const float inv_hf = 1.f / hif;
            const float4 pr = B.rec[q];
            const float4 vi = B.vrec[q];
            const float alpha = S.falpha, beta = S.fbeta, etasq = S.fetasq;
            KahanF ax, ay, ed;
            auto pair = [&](uint32_t code) {
                const uint32_t j = code >> kCodeShift;
                float rabx, raby;  // r_AB = (q - offset) - p from float pairs
                float_pair_rel(S, pr, __ldg(&B.rec[j]), code & 15u, rabx, raby);
                const float d2 = __fmaf_rn(rabx, rabx, raby * raby);
                const float invd = rsqrtf(d2);
                const float qq = fminf(d2 * invd * inv_hf, 1.f);
                const float drk = kdf_f32(S.kernel, qq);
                const float4 vj = __ldg(&B.vrec[j]);
                const float4 dj = __ldg(&D.derf[j]);
                const float vabx = (vj.x - vi.x) + (vj.z - vi.z);
                const float vaby = (vj.y - vi.y) + (vj.w - vi.w);
                const float dot = vabx * rabx + vaby * raby;
                float piab = 0.f;
                if (dot < 0.f) {
                    const float cab = 0.5f * (ci + dj.x);
                    const float rhoab = 0.5f * (rhoi + dj.y);
                    const float hab = 0.5f * (hif + dj.z);
                    // two-instruction quotients (<= 2 ulp; both denominators are
                    // normal: d2 + eta^2 >= eta^2, rho_AB > 0)
                    const float mu = __fdividef(dot * hab, d2 + etasq);
                    piab = __fdividef(mu * (beta * mu - alpha * cab), rhoab);
                }
                const float w = (piab + caf + dj.w) * drk * invd;
                ax.add(rabx * w);
                ay.add(raby * w);
                ed.add(dot * drk);
            };
            for_each_nbr_desc(nb, k, [&](int, uint32_t code) { pair(code); });
            const float ff = S.fdfm * (inv_hf * inv_hf * inv_hf);
            axo = (double)(ax.value_f() * ff) + S.accel[0];
            ayo = (double)(ay.value_f() * ff) + S.accel[1];
            edot = (double)(caf * ed.value_f() * S.fmass);
        }
        if (!is_finite(axo) || !is_finite(ayo) || !is_finite(edot)) fl |= FLAG_Q_RANGE;
        double2 pos = P, vel = B.vel[q];
        double u = B.u[q];
        if (a.integrate) integrate_one(S, pos, vel, u, axo, ayo, edot);
        a.A.pos[q] = pos;
        a.A.vel[q] = vel;
        a.A.u[q] = u;
        a.A.acc[q] = make_double2(axo, ayo);
        a.A.udot[q] = edot;
        a.A.id[q] = B.id[q];
        a.A.hprev[q] = a.D.derf[q].z;  // the smoothing length rounded to FP32
        a.A.vp[q] = B.vp[q];
        a.A.up[q] = B.up[q];
    }
    if (fl) atomicOr(a.c.flags, fl);
}

// The mixed form for few particles: the same arithmetic with the pairs
// dealt over the lanes (pair_tile.cuh). Each pair leaves its factors in shared
// memory, and a lane per particle runs the compensated sums over them,
// farthest first, a term's product fused with the compensation's subtraction
// as in the loop above, so that both kernels return the same bits.
struct MixedRow {
    float4 rec, vrec;  // position and predicted velocity as float pairs
    float inv_h, cterm, h, c, rho;
    int32_t sim;
};

struct MixedWarp {
    float rx[kPairSlots], ry[kPairSlots], w[kPairSlots], dot[kPairSlots], drk[kPairSlots];
    MixedRow row[32];
};

// Kahan's sum with the next term a product: y = x f - c in one rounding
__device__ __forceinline__ void kahan_fma(KahanF &s, float x, float f) {
    const float y = __fmaf_rn(x, f, -s.c);
    const float t = __fadd_rn(s.s, y);
    s.c = __fsub_rn(__fsub_rn(t, s.s), y);
    s.s = t;
}

__global__ void __launch_bounds__(32, kMixedBlocks) k_force_mixed_pairs(ForceArgs a, PairTiles tiles) {
    __shared__ MixedWarp sm;
    const int k = a.c.k, lane = threadIdx.x;
    int W;
    const int64_t q0 = tiles.first(blockIdx.x, W);
    const PArrays &B = a.B;
    const Derived &D = a.D;
    const PairChunks ch(k, W, kPairSlots);
    unsigned fl = 0;
    const int np = (int)min((int64_t)W, a.c.n - q0);
    const int32_t *nb = D.nbr + q0 * k;
    if (lane < np) {
        const int64_t q = q0 + lane;
        const float4 di = D.derf[q];
        MixedRow &R = sm.row[lane];
        R.rec = B.rec[q];
        R.vrec = B.vrec[q];
        R.c = di.x; R.rho = di.y; R.h = di.z; R.cterm = di.w;
        R.inv_h = 1.f / di.z;
        R.sim = sim_of(a.c, q);
    }
    __syncwarp();
    KahanF ax, ay, ed;
    for (int c = 0, e_lo = k; c < ch.n; c++) {
        const int ce = ch.len(c), st = pair_stride(ce), magic = (65535 + ce) / ce, npair = np * ce;
        e_lo -= ce;
        for (int i = lane; i < npair; i += 32) {
            const int p = pair_row(i, magic), at = p * k + e_lo + (i - p * ce), slot = i + p * (st - ce);
            const MixedRow &R = sm.row[p];
            const SimDev &S = a.c.sims[R.sim];
            const uint32_t code = (uint32_t)nb[at], j = code >> kCodeShift;
            const float4 rj = __ldg(&B.rec[j]), vj = __ldg(&B.vrec[j]), dj = __ldg(&D.derf[j]);
            const float4 vi = R.vrec;
            float rabx, raby;  // r_AB = (q - offset) - p from float pairs
            float_pair_rel(S, R.rec, rj, code & 15u, rabx, raby);
            const float d2 = __fmaf_rn(rabx, rabx, raby * raby);
            const float invd = rsqrtf(d2);
            const float qq = fminf(d2 * invd * R.inv_h, 1.f);
            const float drk = kdf_f32(S.kernel, qq);
            const float vabx = (vj.x - vi.x) + (vj.z - vi.z);
            const float vaby = (vj.y - vi.y) + (vj.w - vi.w);
            const float dot = vabx * rabx + vaby * raby;
            float piab = 0.f;
            if (dot < 0.f) {
                const float cab = 0.5f * (R.c + dj.x);
                const float rhoab = 0.5f * (R.rho + dj.y);
                const float hab = 0.5f * (R.h + dj.z);
                // two-instruction quotients (<= 2 ulp; both denominators are
                // normal: d2 + eta^2 >= eta^2, rho_AB > 0)
                const float mu = __fdividef(dot * hab, d2 + S.fetasq);
                piab = __fdividef(mu * (S.fbeta * mu - S.falpha * cab), rhoab);
            }
            sm.rx[slot] = rabx;
            sm.ry[slot] = raby;
            sm.w[slot] = (piab + R.cterm + dj.w) * drk * invd;
            sm.dot[slot] = dot;
            sm.drk[slot] = drk;
        }
        __syncwarp();
        if (lane < np) {
            for (int e = ce - 1; e >= 0; e--) {
                const int t = lane * st + e;
                const float wt = sm.w[t];
                kahan_fma(ax, sm.rx[t], wt);
                kahan_fma(ay, sm.ry[t], wt);
                kahan_fma(ed, sm.dot[t], sm.drk[t]);
            }
        }
        __syncwarp();
    }
    if (lane < np) {
        const int64_t q = q0 + lane;
        const MixedRow &R = sm.row[lane];
        const SimDev &S = a.c.sims[R.sim];
        const float inv_hf = R.inv_h;
        const float ff = S.fdfm * (inv_hf * inv_hf * inv_hf);
        const double axo = (double)(ax.value_f() * ff) + S.accel[0];
        const double ayo = (double)(ay.value_f() * ff) + S.accel[1];
        const double edot = (double)(R.cterm * ed.value_f() * S.fmass);
        if (!is_finite(axo) || !is_finite(ayo) || !is_finite(edot)) fl |= FLAG_Q_RANGE;
        double2 pos = B.pos[q], vel = B.vel[q];
        double u = B.u[q];
        if (a.integrate) integrate_one(S, pos, vel, u, axo, ayo, edot);
        a.A.pos[q] = pos;
        a.A.vel[q] = vel;
        a.A.u[q] = u;
        a.A.acc[q] = make_double2(axo, ayo);
        a.A.udot[q] = edot;
        a.A.id[q] = B.id[q];
        a.A.hprev[q] = R.h;  // the smoothing length rounded to FP32
        a.A.vp[q] = B.vp[q];
        a.A.up[q] = B.up[q];
    }
    if (fl) atomicOr(a.c.flags, fl);
}

// r_AB = (q - offset) - p and v_AB . r_AB for neighbour code `code` of a
// particle at P with predicted velocity vpi (sim/sph.go:355-367)
__device__ __forceinline__ void pair_geom(const SimDev &S, const PArrays &B, uint32_t code, double2 P, double2 vpi,
                                          double &rabx, double &raby, double &dot) {
    const uint32_t j = code >> kCodeShift;
    const double2 vpj = B.vp[j];
    const double vabx = __dsub_rn(vpj.x, vpi.x), vaby = __dsub_rn(vpj.y, vpi.y);
    const double2 Q = B.pos[j];
    if ((code & 15u) == 4u) {  // q - 0 = q exactly
        rabx = __dsub_rn(Q.x, P.x);
        raby = __dsub_rn(Q.y, P.y);
    } else {
        double ox, oy;
        img_shift(S, code & 15u, ox, oy);
        rabx = __dsub_rn(__dsub_rn(Q.x, ox), P.x);
        raby = __dsub_rn(__dsub_rn(Q.y, oy), P.y);
    }
    dot = __dadd_rn(__dmul_rn(vabx, rabx), __dmul_rn(vaby, raby));
}

// ---------------------------------------------------------------- FP64 form.
// A warp takes a tile of W particles (pair_tile.cuh) and, chunk by chunk of
// their lists, farthest first:
//   A. a lane per (particle, entry) pair computes r_AB and v_AB . r_AB, and
//      lists the approaching pairs (v_AB . r_AB < 0) and the others;
//   B. in the listed order, the approaching ones' viscosity terms Pi with all
//      lanes at work (in list order a warp would run them whenever one of its
//      lanes needs them: two divisions, and about half of the pairs), and
//      every pair's terms;
//   C. the ordered sums (sim/sph.go:343-392, farthest first), a lane per
//      particle, or, for tiles of few particles, per particle and component.
// Sums and differences run on the FP64 unit (75 cycles a warp instruction),
// products and quotients on the integer pipes, unchecked behind range tests
// (fp64emu.cuh); pairs that fail one are settled out of line. Every operation and
// its order are the reference's, so the results stay bit-exact.
//
// Zeros fail the range tests, and whole states have them: a lattice or rows
// (r_AB), a state at rest (v_AB), a cold gas (c, and with it cA + cB), viscosity
// off. Out of line they stay on the integer pipes, with the products by zero left
// out; only values outside 2^+-150, infinities, NaNs and coincident particles take
// the hardware's arithmetic. Zero components of r_AB, which lie between others in
// nearly every round, are kept in line: their slot holds kForZero, whose square is
// lost in the other component's, and is marked, and the marked components' terms
// are set to 0 before phase C. Force stage, us, k = 28, with the hardware's
// arithmetic for all of them and so: perfect lattice at rest, N = 250,000, 765 and
// 276 (a jittered moving one 262 both ways), N = 1,048,576 2604 and 749 (949 and
// 953), cold gas moving 2957 and 1048, at rest 3135 and 667, alpha = 0 1602 and
// 1009, viscosity off 1964 and 914. Zero components out of line too: 424 for the
// first; in a form of phase B of its own, for chunks that have them: 0.5 to 2 % more
// for every other state.
//
// Bound (ncu, clustered N = 1,048,576, k = 32): FP64 pipe 73 %, ALU 57 %, issue
// 67 % busy; moving work either way between the two pipes (the sums
// cA + cB, hA + hB, rhoA + rhoB on the integer pipe, the dot product or r^2 on
// the FP64 unit) changed nothing or cost up to 5 %. The loads are issued a
// round early: 1335 -> 1231 us; one loop for both kinds of pairs instead of
// one each: 1231 -> 1160.
//
// Against one warp per 32 particles, a lane each, with the approaching pairs
// compacted per warp (force stage, us): N = 1000 112 -> 14, 10,000 154 -> 29,
// 100,000 297 -> 133 (149 with resident blocks of four warps striding over
// tiles of one width), 1,048,576 1750 -> 1034 (1165), clustered 4,194,304
// 6800 -> 4040 (4540), stress 2,000,003 (k = 64) 6370 -> 3843 (4210).
struct ForceRow {
    double x, y, vx, vy;      // position and predicted velocity
    double c, rho, h, cterm;  // sound speed, density, smoothing length, c^2 / (gamma rho)
};

template <int SLOTS>
struct ForceWarp {
    static_assert(SLOTS % 32 == 0 && pair_rows_fit(SLOTS), "a tile's terms fit its slots at every width");
    double x[SLOTS], y[SLOTS];  // r_AB, then the acceleration terms
    double e[SLOTS];            // v_AB . r_AB, then the du/dt terms
    ForceRow row[32];
    uint16_t list[SLOTS];       // approaching pairs from the front, the others from the back
    uint32_t zx[SLOTS / 32], zy[SLOTS / 32];  // bits of the slots whose x (y) is kForZero
    int marked;                 // the last chunk that has such slots
    __device__ __forceinline__ bool zero_x(int slot) const { return zx[slot >> 5] >> (slot & 31) & 1u; }
    __device__ __forceinline__ bool zero_y(int slot) const { return zy[slot >> 5] >> (slot & 31) & 1u; }
};

// A zero component of r_AB beside one within 2^+-150: its square, 2^-680, lies 380
// binades below the other one's.
constexpr double kForZero = 0x1p-340;

struct Vec2D {
    double x, y;
};

__device__ __forceinline__ bool in_range_or_zero(double x) { return emu_within<150>(x) || emu_is_zero(x); }
__device__ __forceinline__ double emu_halve(double x) { return emu_double(emu_bits(x) - (1ull << 52)); }

// Phase A of a pair that fails its range test: r_AB into the slot, and v_AB . r_AB
// of operands in range or zero, else with hardware arithmetic
template <typename Warp>
__device__ __noinline__ double force_pair_slow(Warp &sm, int slot, int chunk, double rx, double ry, double vx, double vy) {
    const bool mx = emu_is_zero(rx) && emu_within<150>(ry), my = emu_is_zero(ry) && emu_within<150>(rx);
    sm.x[slot] = mx ? kForZero : rx;
    sm.y[slot] = my ? kForZero : ry;
    if (mx) atomicOr(&sm.zx[slot >> 5], 1u << (slot & 31));
    if (my) atomicOr(&sm.zy[slot >> 5], 1u << (slot & 31));
    if (mx || my) sm.marked = chunk;
    if (in_range_or_zero(rx) && in_range_or_zero(ry) && in_range_or_zero(vx) && in_range_or_zero(vy)) {
        const bool zx = emu_is_zero(vx) || emu_is_zero(rx), zy = emu_is_zero(vy) || emu_is_zero(ry);
        if (zx && zy) return 0.0;
        if (zx) return emu_mul_n(vy, ry);
        if (zy) return emu_mul_n(vx, rx);
    }
    return __dadd_rn(__dmul_rn(vx, rx), __dmul_rn(vy, ry));
}

// Pi (sim/sph.go:370-390) from the sums cA + cB, ..., of operands in range or
// zero (cA + cB, alpha, beta), else with hardware arithmetic
__device__ __noinline__ double force_pi_slow(double rx, double ry, double dot, double c2, double rho2, double h2,
                                             double alpha, double beta, double etasq) {
    const bool z1 = emu_is_zero(alpha) || emu_is_zero(c2), z2 = emu_is_zero(beta);
    if (emu_within<350>(rx) && emu_within<350>(ry) && emu_within<400>(dot) && emu_within<150>(rho2) &&
        emu_within<150>(h2) && in_range_or_zero(alpha) && in_range_or_zero(c2) && in_range_or_zero(beta)) {
        const double den = __dadd_rn(__dadd_rn(emu_mul_n(rx, rx), emu_mul_n(ry, ry)), etasq);
        const double mu = emu_div_n(emu_mul_n(dot, emu_halve(h2)), emu_divisor(den));
        if (emu_within<300>(den) && emu_within<300>(mu)) {
            if (z1 && z2) return 0.0;
            const double t1 = z1 ? 0.0 : emu_mul_n(emu_mul_n(emu_neg(alpha), emu_halve(c2)), mu);
            const double t2 = z2 ? 0.0 : emu_mul_n(emu_mul_n(beta, mu), mu);
            const double num = z1 ? t2 : z2 ? t1 : __dadd_rn(t1, t2);
            if (emu_within<800>(num)) return emu_div_n(num, emu_divisor(emu_halve(rho2)));
        }
    }
    const double cab = __dmul_rn(0.5, c2), rhoab = __dmul_rn(0.5, rho2), hab = __dmul_rn(0.5, h2);
    const double r2 = __dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry));
    const double mu = __ddiv_rn(__dmul_rn(dot, hab), __dadd_rn(r2, etasq));
    return __ddiv_rn(__dadd_rn(__dmul_rn(__dmul_rn(-alpha, cab), mu), __dmul_rn(__dmul_rn(beta, mu), mu)), rhoab);
}

struct ForceTerms {
    double x, y, e;
};

// a pair's terms of operands in range or zero, else with hardware arithmetic
template <typename Warp>
__device__ __noinline__ ForceTerms force_terms_slow(const Warp &sm, int slot, double rx, double ry, double dot, double sum3,
                                                    double drk, double d) {
    if (sm.zero_x(slot)) rx = 0.0;
    if (sm.zero_y(slot)) ry = 0.0;
    const bool zd = emu_is_zero(dot) || emu_is_zero(drk), zx = emu_is_zero(rx), zy = emu_is_zero(ry), zs = emu_is_zero(sum3);
    if (in_range_or_zero(rx) && in_range_or_zero(ry) && in_range_or_zero(sum3) && emu_within<150>(d) && in_range_or_zero(drk) &&
        (emu_within<400>(dot) || emu_is_zero(dot))) {
        ForceTerms t{0.0, 0.0, zd ? 0.0 : emu_mul_n(dot, drk)};
        if (zs || emu_is_zero(drk) || (zx && zy)) return t;
        const EmuDivisor dv = emu_divisor(d);
        const double v = emu_div_n(emu_mul_n(emu_mul_n(zx ? ry : rx, sum3), drk), dv);
        if (zx) t.y = v; else t.x = v;
        if (!zx && !zy) t.y = emu_div_n(emu_mul_n(emu_mul_n(ry, sum3), drk), dv);
        return t;
    }
    return ForceTerms{__ddiv_rn(__dmul_rn(__dmul_rn(rx, sum3), drk), d), __ddiv_rn(__dmul_rn(__dmul_rn(ry, sum3), drk), d),
                      __dmul_rn(dot, drk)};
}

template <int SLOTS, int BLOCKS>
__global__ void __launch_bounds__(32, BLOCKS) k_force_fp64(ForceArgs a, PairTiles tiles) {
    __shared__ ForceWarp<SLOTS> sm;
    const int k = a.c.k, lane = threadIdx.x;
    int W;
    const int64_t q0 = tiles.first(blockIdx.x, W);
    const PArrays &B = a.B;
    const Derived &D = a.D;
    const PairChunks ch(k, W, SLOTS);
    unsigned fl = 0;
    const int np = (int)min((int64_t)W, a.c.n - q0);
    const int32_t *nb = D.nbr + q0 * k;
    const double2 *dist = D.dist + q0 * k;
    if (lane < np) {
        const int64_t q = q0 + lane;
        const double2 P = B.pos[q], V = B.vp[q];
        ForceRow &R = sm.row[lane];
        R.x = P.x; R.y = P.y; R.vx = V.x; R.vy = V.y;
        const double4 d = D.der[q];
        R.c = d.x; R.rho = d.y; R.h = d.z; R.cterm = d.w;
    }
    if (lane < SLOTS / 32) sm.zx[lane] = sm.zy[lane] = 0u;
    if (lane == 0) sm.marked = -1;
    __syncwarp();
    double ax = 0.0, ay = 0.0, ed = 0.0;  // (three lanes per particle: ax alone, lane 3 p + component)
    for (int c = 0, e_lo = k; c < ch.n; c++) {
        const int ce = ch.len(c), st = pair_stride(ce), magic = (65535 + ce) / ce, npair = np * ce;
        e_lo -= ce;
        // ---- A
        int nlist = 0, nrest = 0;
        // a round's loads are issued a round (the neighbour's data) or two (its
        // code) before their use
        auto entry = [&](int i) {
            const int p = pair_row(i, magic);
            return p * k + e_lo + (i - p * ce);
        };
        uint32_t code1 = lane < npair ? (uint32_t)nb[entry(lane)] : 0u;
        uint32_t code2 = lane + 32 < npair ? (uint32_t)nb[entry(lane + 32)] : 0u;
        double2 V1 = B.vp[code1 >> kCodeShift], Q1 = B.pos[code1 >> kCodeShift];
        for (int i0 = 0; i0 < npair; i0 += 32) {
            const int i = i0 + lane;
            bool approach = false;
            const uint32_t code = code1;
            const double2 V = V1, Q = Q1;
            code1 = code2;
            V1 = B.vp[code1 >> kCodeShift];
            Q1 = B.pos[code1 >> kCodeShift];
            code2 = i + 64 < npair ? (uint32_t)nb[entry(i + 64)] : 0u;
            if (i < npair) {
                const int p = pair_row(i, magic), slot = i + p * (st - ce);
                const ForceRow &R = sm.row[p];
                const double vx = __dsub_rn(V.x, R.vx), vy = __dsub_rn(V.y, R.vy);
                double qx = Q.x, qy = Q.y;
                if ((code & 15u) != 4u) {
                    double ox, oy;
                    img_shift(a.c.sims[sim_of(a.c, q0 + p)], code & 15u, ox, oy);
                    qx = __dsub_rn(qx, ox);
                    qy = __dsub_rn(qy, oy);
                }
                const double rx = __dsub_rn(qx, R.x), ry = __dsub_rn(qy, R.y);
                double dot;
                if (emu_within<150>(rx) && emu_within<150>(ry) && emu_within<150>(vx) && emu_within<150>(vy)) {
                    dot = __dadd_rn(emu_mul_n(vx, rx), emu_mul_n(vy, ry));  // 0, or 2^-353 at least (no subnormal)
                    approach = emu_hi(dot) > 0x80000000u;
                    sm.x[slot] = rx;
                    sm.y[slot] = ry;
                } else {
                    dot = force_pair_slow(sm, slot, c, rx, ry, vx, vy);
                    approach = emu_bits(dot) > kEmuSign && !is_nan(dot);
                }
                sm.e[slot] = dot;
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, approach);
            const int before = __popc(bal & lanemask_lt());
            if (i < npair) sm.list[approach ? nlist + before : npair - 1 - (nrest + lane - before)] = (uint16_t)i;
            nlist += __popc(bal);
            nrest = min(i0 + 32, npair) - nlist;
        }
        __syncwarp();
        // ---- B, the approaching pairs first: one round at most holds both kinds
        int at = lane < npair ? entry(sm.list[lane]) : 0;
        double2 dd1 = dist[at];  // (NNDists, dF)
        const double4 *der1 = D.der + ((uint32_t)nb[at] >> kCodeShift);  // (c, rho, h, c^2 / (gamma rho))
        double c1 = 0.0, rho1 = 0.0, h1 = 0.0, ct1 = der1->w;
        if (lane < nlist) { c1 = der1->x; rho1 = der1->y; h1 = der1->z; }
        for (int n = lane; n < npair; n += 32) {
            const double2 dd = dd1;
            const double cj = c1, rhoj = rho1, hj = h1, ctj = ct1;
            if (n + 32 < npair) {
                at = entry(sm.list[n + 32]);
                dd1 = dist[at];
                der1 = D.der + ((uint32_t)nb[at] >> kCodeShift);
                ct1 = der1->w;
                if (n + 32 < nlist) { c1 = der1->x; rho1 = der1->y; h1 = der1->z; }
            }
            const int i = sm.list[n], p = pair_row(i, magic), slot = i + p * (st - ce);
            const ForceRow &R = sm.row[p];
            const double rx = sm.x[slot], ry = sm.y[slot], dot = sm.e[slot];
            const bool in_r = emu_within<350>(rx) && emu_within<350>(ry);  // (kForZero included; the products below stay normal)
            double sum = R.cterm;  // Pi + cA (0 + cA = cA)
            if (n < nlist) {
                const SimDev &S = a.c.sims[sim_of(a.c, q0 + p)];
                const double alpha = S.alpha, beta = S.beta;
                const double c2 = __dadd_rn(R.c, cj), rho2 = __dadd_rn(R.rho, rhoj), h2 = __dadd_rn(R.h, hj);
                bool ok = in_r && emu_within<400>(dot) && emu_within<150>(c2) && emu_within<150>(rho2) &&
                          emu_within<150>(h2) && emu_within<150>(alpha) && emu_within<150>(beta);
                double pi = 0.0;
                if (ok) {
                    const double den = __dadd_rn(__dadd_rn(emu_mul_n(rx, rx), emu_mul_n(ry, ry)), S.etasq);
                    const double mu = emu_div_n(emu_mul_n(dot, emu_halve(h2)), emu_divisor(den));
                    const double num = __dadd_rn(emu_mul_n(emu_mul_n(emu_neg(alpha), emu_halve(c2)), mu),
                                                 emu_mul_n(emu_mul_n(beta, mu), mu));
                    pi = emu_div_n(num, emu_divisor(emu_halve(rho2)));
                    ok = emu_within<300>(den) && emu_within<300>(mu) && emu_within<800>(num);
                }
                if (!ok) pi = force_pi_slow(rx, ry, dot, c2, rho2, h2, alpha, beta, S.etasq);
                sum = __dadd_rn(pi, sum);
            }
            // the terms r_AB (Pi + cA + cB) dF / NNDists and v_AB . r_AB dF
            sum = __dadd_rn(sum, ctj);
            const double d = dd.x, drk = dd.y;
            // a zero dF (always so for the farthest neighbour) makes zero terms, whose
            // signs do not matter to the sums, which are never -0
            const bool dz = emu_is_zero(drk), dot0 = emu_is_zero(dot);
            ForceTerms t;
            if (in_r && emu_within<150>(sum) && emu_within<150>(d) && (dz || emu_within<150>(drk)) &&
                (emu_within<400>(dot) || dot0)) {
                const EmuDivisor dv = emu_divisor(d);  // shared by both quotients
                t.x = emu_div_n(emu_mul_n(emu_mul_n(rx, sum), drk), dv);
                t.y = emu_div_n(emu_mul_n(emu_mul_n(ry, sum), drk), dv);
                t.e = emu_mul_n(dot, drk);
                if (dz) t.x = t.y = 0.0;
                if (dz || dot0) t.e = 0.0;
            } else {
                t = force_terms_slow(sm, slot, rx, ry, dot, sum, drk, d);
            }
            sm.x[slot] = t.x;
            sm.y[slot] = t.y;
            sm.e[slot] = t.e;
        }
        __syncwarp();
        if (sm.marked == c) {  // the marked components' terms (0 times a NaN or an infinity stays)
            for (int slot = lane; slot < np * st; slot += 32) {
                if (sm.zero_x(slot) && !is_nan(sm.x[slot])) sm.x[slot] = 0.0;
                if (sm.zero_y(slot) && !is_nan(sm.y[slot])) sm.y[slot] = 0.0;
            }
            __syncwarp();
            if (lane < SLOTS / 32) sm.zx[lane] = sm.zy[lane] = 0u;
        }
        // ---- C
        if (W <= kSplitWidth) {
            if (lane < 3 * np) {
                const int p = lane / 3, comp = lane - 3 * p;
                const double *t = (comp == 0 ? sm.x : comp == 1 ? sm.y : sm.e) + p * st;
                for (int e = ce - 1; e >= 0; e--) ax = __dadd_rn(ax, t[e]);
            }
        } else if (lane < np) {
            const int t = lane * st;
            for (int e = ce - 1; e >= 0; e--) {
                ax = __dadd_rn(ax, sm.x[t + e]);
                ay = __dadd_rn(ay, sm.y[t + e]);
                ed = __dadd_rn(ed, sm.e[t + e]);
            }
        }
        __syncwarp();
    }
    if (W <= kSplitWidth) {
        const double s = ax;
        const int l3 = min(3 * lane, 29);
        ax = __shfl_sync(0xffffffffu, s, l3);
        ay = __shfl_sync(0xffffffffu, s, l3 + 1);
        ed = __shfl_sync(0xffffffffu, s, l3 + 2);
    }
    if (lane < np) {
        const int64_t q = q0 + lane;
        const ForceRow &R = sm.row[lane];
        const SimDev &S = a.c.sims[sim_of(a.c, q)];
        const double hi = R.h;
        const double h3 = emu_mul(emu_mul(hi, hi), hi);
        const double f = emu_div(emu_mul(S.mass, S.dfpref), emu_divisor(h3), h3);
        const double axo = __dadd_rn(emu_mul(ax, f), S.accel[0]);
        const double ayo = __dadd_rn(emu_mul(ay, f), S.accel[1]);
        const double edot = emu_mul(emu_mul(R.cterm, ed), S.mass);
        if (!is_finite(axo) || !is_finite(ayo) || !is_finite(edot)) fl |= FLAG_Q_RANGE;
        double2 pos = make_double2(R.x, R.y), vel = B.vel[q];
        double u = B.u[q];
        if (a.integrate) integrate_one(S, pos, vel, u, axo, ayo, edot);
        a.A.pos[q] = pos;
        a.A.vel[q] = vel;
        a.A.u[q] = u;
        a.A.acc[q] = make_double2(axo, ayo);
        a.A.udot[q] = edot;
        a.A.id[q] = B.id[q];
        a.A.hprev[q] = (float)hi;
        a.A.vp[q] = make_double2(R.vx, R.vy);
        a.A.up[q] = B.up[q];
    }
    if (fl) atomicOr(a.c.flags, fl);
}

// resident blocks (warps) per SM of a form of the FP64 force
template <int SLOTS, int BLOCKS>
static int force_blocks() {
    static const int per_sm = [] {
        int nb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_force_fp64<SLOTS, BLOCKS>, 32, 0);
        return std::max(nb, 1);
    }();
    return per_sm;
}

template <int SLOTS, int BLOCKS>
static void launch_force_fp64(const ForceArgs &a, const Launch &L) {
    const PairTiles t(a.c.n, L.sms, force_blocks<SLOTS, BLOCKS>(), kForceNarrow);
    k_force_fp64<SLOTS, BLOCKS><<<t.grid(), 32, 0, L.stream>>>(a, t);
}

void launch_force(const Ctx &c, const Launch &L, const PArrays &B, const PArrays &A,
                  const Derived &D, int mode, bool integrate) {
    ForceArgs a;
    a.c = c;
    a.B = B;
    a.A = A;
    a.D = D;
    a.integrate = integrate ? 1 : 0;
    if (mode != MODE_MIXED) {
        const int64_t pass1 = 32ll * L.sms * force_blocks<kPairSlots, kForceBlocks>();
        const int64_t pass2 = 32ll * L.sms * force_blocks<kForceSlotsMany, kForceBlocksMany>();
        const bool wide = c.n <= pass2 || (2 * c.n > 3 * pass2 && 10 * c.n <= 21 * pass1);
        if (wide) launch_force_fp64<kPairSlots, kForceBlocks>(a, L);
        else launch_force_fp64<kForceSlotsMany, kForceBlocksMany>(a, L);
        return;
    }
    if (c.n <= kMixedPairsMaxN) {
        const PairTiles t(c.n, L.sms, kMixedBlocks, kForceNarrow);
        k_force_mixed_pairs<<<t.grid(), 32, 0, L.stream>>>(a, t);
        return;
    }
    k_force_mixed<<<(int)((c.n + 127) / 128), 128, 0, L.stream>>>(a);
}

// ------------------------------------------------------------ error norms
// Per particle, the sums of the magnitudes of its neighbour terms in the
// acceleration and in du/dt: the normalisers of the mixed form's error
// statements. Read from the FP64 form's last evaluation (positions, predicted
// velocities, lists with (NNDists, dF), per-particle (c, rho, h, c^2/(gamma
// rho))), in the reference's term order (sim/sph.go:343-392, farthest first)
// and rounding, so that they equal the oracle's norms bit for bit.
__global__ void k_error_norms(Ctx c, PArrays B, Derived D, double *anorm, double *unorm) {
    const int k = c.k;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < c.n;
         q += (int64_t)gridDim.x * blockDim.x) {
        const SimDev &S = c.sims[sim_of(c, q)];
        const double2 P = B.pos[q], vpi = B.vp[q];
        const double4 di = D.der[q];  // (c, rho, h, c^2/(gamma rho))
        const int32_t *nb = D.nbr + q * k;
        const double2 *dist = D.dist + q * k;
        double an = 0.0, un = 0.0;
        for (int e = k - 1; e >= 0; e--) {
            const uint32_t code = (uint32_t)nb[e];
            double rabx, raby, dot;
            pair_geom(S, B, code, P, vpi, rabx, raby, dot);
            const double d = dist[e].x, drk = dist[e].y;
            const double4 dj = D.der[code >> kCodeShift];
            double piab = 0.0;
            if (dot < 0.0) {
                const double cab = __dmul_rn(0.5, __dadd_rn(di.x, dj.x));
                const double rhoab = __dmul_rn(0.5, __dadd_rn(di.y, dj.y));
                const double hab = __dmul_rn(0.5, __dadd_rn(di.z, dj.z));
                const double r2 = __dadd_rn(__dmul_rn(rabx, rabx), __dmul_rn(raby, raby));
                const double mu = __ddiv_rn(__dmul_rn(dot, hab), __dadd_rn(r2, S.etasq));
                piab = __ddiv_rn(__dadd_rn(__dmul_rn(__dmul_rn(-S.alpha, cab), mu), __dmul_rn(__dmul_rn(S.beta, mu), mu)),
                                 rhoab);
            }
            const double w = __ddiv_rn(__dmul_rn(__dadd_rn(__dadd_rn(piab, di.w), dj.w), drk), d);
            an = __dadd_rn(an, __dmul_rn(__dsqrt_rn(__dadd_rn(__dmul_rn(rabx, rabx), __dmul_rn(raby, raby))), fabs(w)));
            un = __dadd_rn(un, fabs(__dmul_rn(dot, drk)));
        }
        const double f = __ddiv_rn(__dmul_rn(S.mass, S.dfpref), __dmul_rn(__dmul_rn(di.z, di.z), di.z));
        const int32_t id = B.id[q];
        anorm[id] = __dmul_rn(an, fabs(f));
        unorm[id] = __dmul_rn(un, fabs(__dmul_rn(di.w, S.mass)));
    }
}

void launch_error_norms(const Ctx &c, const Launch &L, const PArrays &B, const Derived &D, double *anorm,
                        double *unorm) {
    const int block = 256;
    const int64_t need = (c.n + block - 1) / block;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)L.sms * 8));
    k_error_norms<<<grid, block, 0, L.stream>>>(c, B, D, anorm, unorm);
}

}  // namespace sphgpu
