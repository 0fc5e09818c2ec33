// k_density.cu -- smoothing length, density (sim/sph.go:306-323), sound speed
// (sim/sph.go:421-429) and c^2/(gamma rho) of the FP64 forms, in the
// reference's operation order and rounding, and dF(q) per neighbour for the
// force.
//
// Per neighbour: the squared distance in the reference's rounding, its square
// root, q = d/h, the kernel F(q) and its derivative, one addition to the
// ordered sum. An FP64 instruction holds a sub-partition's FP64 unit for 75
// cycles, and an integer instruction its ALU for two, so the differences and
// sums run in hardware (four per pair, three more where q < 1/2) and the
// products, quotients and roots on the integer pipes (fp64emu.cuh), unchecked
// behind one range test per pair; pair_slow computes a pair that fails it with
// the hardware alone. ncu, clustered N = 1,048,576, k = 32: FP64 pipe 67 %, ALU
// 67 %, issue 70 % busy, none of them alone the bound; the next round's loads
// issued early changed nothing.
//
// Measured against one thread per particle with three passes over its list
// (density stage, us): N = 1000 49 -> 12, 10,000 61 -> 21, 100,000 107 -> 70,
// 1,048,576 690 -> 502 (540 with resident blocks of four warps striding over
// the tiles), clustered 4,194,304 2620 -> 1893 (2190).
#include "pair_tile.cuh"

#include <algorithm>

namespace sphgpu {

namespace {

constexpr int kDensityNarrow = 10;

struct DensityArgs {
    Ctx c;
    PArrays B;
    Derived D;
    PairTiles tiles;
};

// what the pairs of a particle share: its position, h and h as a divisor
struct alignas(16) DensityRow {
    double x, y, h;
    uint64_t mb, inv;
    int32_t kernel;  // with its image shifts, the only per-simulation data a pair reads
    int32_t sim;
};

static_assert(pair_rows_fit(kPairSlots), "a tile's terms fit its slots at every width");

struct DensityWarp {
    DensityRow row[32];
    double term[kPairSlots];   // F(q) of the chunk's pairs (q itself for those waiting in near)
    uint16_t near[kPairSlots]; // pairs with q < 1/2 (Monahan)
};

struct PairF {
    double d, f, df;
};

// The distance of two particles on a common row or column, whose zero
// difference the unchecked product does not take: the other difference's
// magnitude, since RN(sqrt(RN(y^2))) = |y| in binary arithmetic within the range.
// (S. Boldo, "Stupid is as stupid does: taking the square root of the square of a
// floating-point number", 2015.) 0 where neither difference is zero, or both.
// Lattices and rows have such pairs in nearly every round; with them left to
// pair_slow a round paid for its hardware root, quotient and kernel function
// (density stage of a perfect lattice, N = 1,048,576, k = 28: 1826 us, so 539; a
// jittered one 448 both ways). As an operand in the zero's place instead, 456, but
// 2.5 % on every other state; out of line, 452 and 0.4 %.
__device__ __forceinline__ double axis_distance(double dx, double dy) {
    const double a = emu_is_zero(dx) ? dy : emu_is_zero(dy) ? dx : 0.0;
    return emu_double(emu_bits(a) & ~kEmuSign);
}

// One pair with hardware arithmetic: operands the unchecked integer
// operations do not take (coincident particles, values outside 2^+-150,
// infinities and NaNs).
__device__ __noinline__ PairF pair_slow(double dx, double dy, double h, int kernel) {
    PairF r;
    r.d = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    const double q = __ddiv_rn(r.d, h);
    r.f = kf_exact(kernel, q);
    r.df = kdf_exact(kernel, q);
    return r;
}

// F and dF of the Monahan kernel for q in [1/2, 1): (1 - q)^3 / 3 and
// -(1 - q)^2, the difference exact
__device__ __forceinline__ void monahan_far(double q, PairF &r) {
    const double z = emu_one_minus_n(q);
    const double z2 = emu_mul_n(z, z);
    r.f = emu_div3_n(emu_mul_n(z2, z));
    r.df = emu_neg(z2);
}

// for q < 1/2: q^3 - q^2 + 1/6 and 3 q^2 - 2 q
__device__ __forceinline__ void monahan_near(double q, double &f, double &df) {
    const double q2 = emu_mul_n(q, q);
    f = __dadd_rn(__dsub_rn(emu_mul_n(q2, q), q2), 1.0 / 6.0);
    df = __dsub_rn(emu_mul_n(emu_mul_n(3.0, q), q), emu_double(emu_bits(q) + (1ull << 52)));
}

__device__ __forceinline__ void wendland(double q, PairF &r) {
    const double a = __dsub_rn(1.0, q);
    const double t = emu_mul_n(emu_mul_n(emu_mul_n(a, a), a), a);
    r.f = emu_mul_n(t, __dadd_rn(1.0, emu_double(emu_bits(q) + (2ull << 52))));
    r.df = emu_mul_n(emu_mul_n(emu_mul_n(__dmul_rn(-10.0, q), a), a), a);
}

// 32 blocks (64 registers): 502 us at N = 1,048,576 against 510 to 512 at 20,
// 24 and 28 (no spills either)
__global__ void __launch_bounds__(32, 32) k_density_fp64(DensityArgs a) {
    __shared__ DensityWarp sm;
    const int k = a.c.k, lane = threadIdx.x;
    const PArrays &B = a.B;
    int W;
    const int64_t q0 = a.tiles.first(blockIdx.x, W);
    const PairChunks ch(k, W, kPairSlots);
    unsigned fl = 0;
    const int np = (int)min((int64_t)W, a.c.n - q0);
    const int32_t *nb = a.D.nbr + q0 * k;
    double2 *dist = a.D.dist + q0 * k;
    double h = 1.0, acc = 0.0;
    if (lane < np) {
        const int s = sim_of(a.c, q0 + lane);
        const SimDev &S = a.c.sims[s];
        const double2 P = B.pos[q0 + lane];
        const double dk2 = nbr_d2(S, B, P, (uint32_t)nb[lane * k + k - 1]);
        if (!(dk2 < 0.4)) fl |= FLAG_SENTINEL;
        h = emu_sqrt(dk2);
        const EmuDivisor dh = emu_divisor(h);  // shared by the k quotients d/h
        DensityRow &R = sm.row[lane];
        R.x = P.x;
        R.y = P.y;
        R.h = h;
        R.mb = dh.mb;
        R.inv = dh.inv;
        R.kernel = S.kernel;
        R.sim = s;
    }
    const bool plain = __all_sync(0xffffffffu, emu_within<150>(h));
    __syncwarp();
    for (int c = 0, e_lo = k; c < ch.n; c++) {
        const int ce = ch.len(c), st = pair_stride(ce), magic = (65535 + ce) / ce;
        e_lo -= ce;
        int nnear = 0;
        for (int i0 = 0; i0 < np * ce; i0 += 32) {
            const int i = i0 + lane;
            bool near = false;
            int slot = 0;
            if (i < np * ce) {
                const int p = pair_row(i, magic), at = p * k + e_lo + (i - p * ce);
                slot = i + p * (st - ce);
                const DensityRow &R = sm.row[p];
                const uint32_t code = (uint32_t)nb[at];
                const double2 Q = B.pos[code >> kCodeShift];
                double px = R.x, py = R.y;
                if ((code & 15u) != 4u) {
                    double ox, oy;
                    img_shift(a.c.sims[R.sim], code & 15u, ox, oy);
                    px = __dadd_rn(px, ox);
                    py = __dadd_rn(py, oy);
                }
                const double dx = __dsub_rn(px, Q.x), dy = __dsub_rn(py, Q.y);
                PairF r;
                bool in = plain && emu_within<150>(dx) && emu_within<150>(dy);
                if (in) {
                    r.d = emu_sqrt_n(__dadd_rn(emu_mul_n(dx, dx), emu_mul_n(dy, dy)));
                } else {
                    r.d = axis_distance(dx, dy);
                    in = plain && emu_within<150>(r.d);
                }
                if (in) {
                    const double q = emu_div_n(r.d, EmuDivisor{R.mb, R.inv, emu_hi(R.h)});  // in (0, 1]: d <= h
                    const uint32_t qh = emu_hi(q);
                    near = R.kernel != SPH_KERNEL_WENDLAND && qh < 0x3fe00000u;
                    if (near) r.f = q;
                    else if (R.kernel != SPH_KERNEL_WENDLAND) monahan_far(q, r);
                    else wendland(q, r);
                    if (qh == 0x3ff00000u) {  // q = 1: 1 - q = 0, which the products do not take
                        r.f = 0.0;
                        r.df = -0.0;
                    }
                } else {
                    r = pair_slow(dx, dy, R.h, R.kernel);
                }
                dist[at] = make_double2(r.d, r.df);
                sm.term[slot] = r.f;
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, near);
            if (near) sm.near[nnear + __popc(bal & lanemask_lt())] = (uint16_t)i;
            nnear += __popc(bal);
        }
        __syncwarp();
        // the pairs with q < 1/2, with all lanes at work (a quarter of the
        // pairs, but some of them in half of the rounds above)
        for (int n = lane; n < nnear; n += 32) {
            const int i = sm.near[n], p = pair_row(i, magic), slot = i + p * (st - ce);
            double f, df;
            monahan_near(sm.term[slot], f, df);
            sm.term[slot] = f;
            dist[p * k + e_lo + (i - p * ce)].y = df;
        }
        __syncwarp();
        if (lane < np) {
            const double *t = sm.term + lane * st;
            for (int e = ce - 1; e >= 0; e--) acc = __dadd_rn(acc, t[e]);
        }
        __syncwarp();
    }
    if (lane < np) {
        const int64_t q = q0 + lane;
        const SimDev &S = a.c.sims[sim_of(a.c, q)];
        const double gamma = S.gamma, up = B.up[q];
        const double hh = emu_mul(h, h);
        const double rho = emu_div(emu_mul(__dmul_rn(S.fpref, S.mass), acc), emu_divisor(hh), hh);
        if (!(rho >= 0.0 && rho < 1.0e308)) fl |= FLAG_Q_RANGE;  // a NaN or infinite distance
        const double cs = emu_sqrt(emu_mul(__dmul_rn(gamma, __dsub_rn(gamma, 1.0)), up));
        const double grho = emu_mul(gamma, rho);
        const double ct = emu_div(emu_mul(cs, cs), emu_divisor(grho), grho);
        a.D.rho[q] = rho;
        a.D.c[q] = cs;
        a.D.h[q] = h;
        a.D.der[q] = make_double4(cs, rho, h, ct);
    }
    if (fl) atomicOr(a.c.flags, fl);
}

}  // namespace

void launch_density_fp64(const Ctx &c, const Launch &L, const PArrays &B, const Derived &D) {
    static const int per_sm = [] {
        int nb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_density_fp64, 32, 0);
        return std::max(nb, 1);
    }();
    DensityArgs a{c, B, D, PairTiles(c.n, L.sms, per_sm, kDensityNarrow)};
    k_density_fp64<<<a.tiles.grid(), 32, 0, L.stream>>>(a);
}

}  // namespace sphgpu
