// fp64emu.cuh -- binary64 multiplication, addition, subtraction, division
// and square root, rounded to nearest with ties to even (IEEE 754-2019,
// 4.3.1), and the split of a binary64 into a float pair, computed with
// integer instructions (and FP32 seeds and conversions).
//
// GB300 issues two FP64 lanes per SM per clock: one warp-wide FP64
// instruction holds a sub-partition's FP64 unit for 75 cycles (measured), while
// the same sub-partition can issue one instruction of another kind every
// cycle. So the FP64 kernels compute products, quotients and roots here, on
// the integer and FP32 pipes, beside the hardware's additions (their FP64 unit,
// ALU and issue slots are then each about two thirds busy). Every result is the
// hardware instruction's, bit for bit (sph_selftest_fp64emu checks each, and the
// unchecked forms over the ranges that the kernels' tests admit, against
// __dmul_rn, __dadd_rn, __dsub_rn, __ddiv_rn, __dsqrt_rn and the double -> float
// conversion). The checked sum, difference and 1 - x are called by these checks
// alone at present.
//
// Method for products and sums (the textbook guard digits and sticky bit,
// e.g. D. Goldberg, "What every computer scientist should know about
// floating-point arithmetic", ACM Computing Surveys 23(1), 1991; quotients
// and square roots are described at their functions):
//   * product: the exact 106-bit product of the two 53-bit significands, its
//     leading 53 bits rounded on the remaining bits (round bit, then "any
//     bit below it" as the sticky);
//   * sum: significands left-aligned with 10 guard bits, the smaller one
//     shifted right by the exponent difference with the shifted-out bits
//     jammed into its lowest bit, added or subtracted exactly, normalised,
//     rounded on the guard bits.
// Operands or results outside the normal range (zeros in a product,
// subnormals, infinities, NaNs, overflow in a sum, underflow) and sums of
// operands more than 63 binades apart take the hardware instruction, so
// those rare cases need no integer code at all.
// That instruction sits in a function that is never inlined, behind a
// branch: a fallback the compiler could compute speculatively (and select)
// would occupy the FP64 unit on every call (measured: the emulated product
// then ran no faster than the hardware's).
#pragma once
#include <stdint.h>

namespace sphgpu {

static __device__ __noinline__ double emu_native_mul(double x, double y) { return __dmul_rn(x, y); }
static __device__ __noinline__ double emu_native_add(double x, double y) { return __dadd_rn(x, y); }
static __device__ __noinline__ double emu_native_sub(double x, double y) { return __dsub_rn(x, y); }
static __device__ __noinline__ double emu_native_sqrt(double x) { return __dsqrt_rn(x); }
static __device__ __noinline__ double emu_native_div(double x, double y) { return __ddiv_rn(x, y); }

constexpr uint64_t kEmuSign = 0x8000000000000000ull;
constexpr uint64_t kEmuFrac = 0x000FFFFFFFFFFFFFull;
constexpr uint64_t kEmuHidden = 0x0010000000000000ull;

__device__ __forceinline__ uint64_t emu_bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double emu_double(uint64_t b) { return __longlong_as_double((long long)b); }

// ---- words and carries. The device forms are PTX (a carry chain, a left
// funnel shift, the approximate FP32 seeds); the host forms serve the
// host-compiled check of the same arithmetic.
__device__ __forceinline__ uint32_t emu_hi(double x) { return (uint32_t)(emu_bits(x) >> 32); }
__device__ __forceinline__ uint32_t emu_lo(double x) { return (uint32_t)emu_bits(x); }

// -x (the compiler negates a double with an FP64 instruction)
__device__ __forceinline__ double emu_neg(double x) { return emu_double(emu_bits(x) ^ kEmuSign); }

// the high word of (hi:lo) << s, s in 0 .. 31
__device__ __forceinline__ uint32_t emu_fsl(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31u)) >> 32);
#endif
}

__device__ __forceinline__ float emu_rcp_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}

__device__ __forceinline__ float emu_rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return rsqrtf(x);
#endif
}

// The double (hi:lo) rounded up when the bits below it, (r1:r0), exceed half
// a unit, or equal it and lo is odd: the carry out of (r1 : r0 | odd) +
// (2^63 - 1) is exactly that decision, and runs on into the exponent when the
// significand overflows.
__device__ __forceinline__ double emu_round_pack(uint32_t hi, uint32_t lo, uint32_t r1, uint32_t r0) {
    r0 |= lo & 1u;
#ifdef __CUDA_ARCH__
    uint32_t ol, oh;
    asm("{\n\t.reg .u32 t;\n\t"
        "add.cc.u32 t, %2, 0xffffffff;\n\t"
        "addc.cc.u32 t, %3, 0x7fffffff;\n\t"
        "addc.cc.u32 %0, %4, 0;\n\t"
        "addc.u32 %1, %5, 0;\n\t}"
        : "=r"(ol), "=r"(oh)
        : "r"(r0), "r"(r1), "r"(lo), "r"(hi));
    return emu_double(((uint64_t)oh << 32) | ol);
#else
    const uint64_t r = ((uint64_t)r1 << 32) | r0;
    return emu_double((((uint64_t)hi << 32) | lo) + (r > 0x8000000000000000ull ? 1ull : 0ull));
#endif
}

// ---- the operations without their range checks: operands normal (not zero,
// subnormal, infinite or NaN) and the result's exponent in the normal range,
// both the caller's to ensure.

// RN(x y): the 106-bit product of the significands from four 32 x 32 ->
// 64-bit products, its leading 53 bits and the two words below them by funnel
// shifts. 40 cycles per warp and sub-partition in a probe of independent
// chains, against 75 for the hardware's DMUL and 61 for the form this
// replaced (the round and sticky bits extracted and compared). Two variants
// that moved the alignment and the normalisation to the multiply pipe
// (multiplications by powers of two) took 53 to 55: the 64-bit addends they
// zero-extend cost register moves.
__device__ __forceinline__ double emu_mul_n(double x, double y) {
    const uint32_t xh = emu_hi(x), a0 = emu_lo(x), yh = emu_hi(y), b0 = emu_lo(y);
    const uint32_t a1 = (xh & 0xfffffu) | 0x100000u, b1 = (yh & 0xfffffu) | 0x100000u;
    const uint64_t t0 = (uint64_t)a0 * b0;
    const uint64_t m = (uint64_t)a0 * b1 + (uint64_t)a1 * b0 + (t0 >> 32);  // < 2^55
    const uint64_t u = (uint64_t)a1 * b1 + (m >> 32);
    const uint32_t w0 = (uint32_t)t0, w1 = (uint32_t)m, w2 = (uint32_t)u, w3 = (uint32_t)(u >> 32);
    const uint32_t top = w3 >> 9, sh = 20u + top;  // product >= 2: the significand is its bits from 53 on, else from 52
    // sign and exponent: the sum's carry out of the sign bits is their XOR;
    // the hidden bit (and a rounding carry) add one
    const uint32_t eh = (xh & 0xfff00000u) + (yh & 0xfff00000u) + ((top << 20) - (1024u << 20));
    return emu_round_pack(__funnelshift_r(w2, w3, sh) + eh, __funnelshift_r(w1, w2, sh), __funnelshift_r(w0, w1, sh),
                          __funnelshift_r(0u, w0, sh));
}

// Whether |x| lies in [2^-L, 2^L): one multiply-add and one compare, the sign
// shifted out. False for zeros, infinities and NaNs.
template <uint32_t L>
__device__ __forceinline__ bool emu_within(double x) {
    return emu_hi(x) * 2u - ((1023u - L) << 21) < (2u * L) << 21;
}

__device__ __forceinline__ bool emu_is_zero(double x) { return ((emu_hi(x) * 2u) | emu_lo(x)) == 0u; }

// RN(x y): the unchecked product, or the hardware's when an operand lies
// outside [2^-500, 2^500) (zeros, subnormals, infinities and NaNs included)
__device__ __forceinline__ double emu_mul(double x, double y) {
    double r = emu_mul_n(x, y);
    if (!(emu_within<500>(x) && emu_within<500>(y))) r = emu_native_mul(x, y);
    return r;
}

// RN(x x): as emu_mul, but a zero, which differences of coordinates on a lattice
// often are, squares without the hardware
__device__ __forceinline__ double emu_sq(double x) {
    double r = emu_mul_n(x, x);
    if (!emu_within<500>(x)) r = emu_is_zero(x) ? 0.0 : emu_native_mul(x, x);
    return r;
}

// u as a float, truncated
__device__ __forceinline__ float emu_u2f_rz(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint2float_rz(u);
#else
    const int lz = u ? __builtin_clz(u) : 0;
    return (float)(lz < 8 ? u & ~((1u << (8 - lz)) - 1u) : u);
#endif
}

// 1 - x for x in [1/2, 1), where the difference is exact (Sterbenz):
// 1 - x = t 2^-53 with t = 2^53 - m for the significand m of x, shifted to put
// its leading bit at bit 52. The leading bit comes from the exponent of t's
// top 32 bits as a float (a conversion issues four times as often as a count
// of leading zeros: 20 cycles in the probe against 57); x closer to 1 than
// 2^-32 takes the hardware subtraction.
__device__ __forceinline__ double emu_one_minus_n(double x) {
    const uint64_t t = (1ull << 53) - ((emu_bits(x) & kEmuFrac) | kEmuHidden);  // (0, 2^52]
    const uint32_t tl = (uint32_t)t, th = (uint32_t)(t >> 32);
    const uint32_t top = emu_fsl(tl, th, 11);  // t >> 21
    const uint32_t lz = 158u - (__float_as_uint(emu_u2f_rz(top)) >> 23);  // 0 .. 31
    double r = emu_double(((uint64_t)(emu_fsl(tl, th, lz) + ((1021u - lz) << 20)) << 32) | (tl << (lz & 31u)));
    if (top == 0u) r = emu_native_sub(1.0, x);
    return r;
}

// RN(1 - x): the unchecked difference, or the hardware's for x outside [1/2, 1)
__device__ __forceinline__ double emu_one_minus(double x) {
    double r = emu_one_minus_n(x);
    if (emu_hi(x) >> 20 != 1022u) r = emu_native_sub(1.0, x);
    return r;
}

static __device__ __noinline__ float emu_native_d2f(double x) { return __double2float_rn(x); }

// RN_float(v): the significand rounded to 24 bits, ties to even. (The
// hardware's conversion holds the FP64 unit as long as an addition.) Values
// whose float would not be normal take it.
__device__ __forceinline__ float emu_d2f(double v) {
    const uint32_t ah = emu_hi(v), al = emu_lo(v);
    const uint32_t e = (ah >> 20) & 0x7ffu;
    const uint32_t q = emu_fsl(al, (ah & 0xfffffu) | 0x100000u, 3), rem = al & 0x1fffffffu;  // q: 24 bits
    const uint32_t up = rem + (q & 1u) > 0x10000000u ? 1u : 0u;
    float f = __uint_as_float((ah & 0x80000000u) | (((e - 897u) << 23) + q + up));
    if (!(e - 897u < 253u)) f = emu_native_d2f(v);
    return f;
}

// The float pair of v: hi = RN_float(v) and lo = RN_float(v - hi) (v - hi is
// exact in binary64). hi rounds the 53-bit significand to 24 bits; the
// remainder t = m - hi's significand 2^29 is an integer below 2^29 in
// magnitude, converted by the FP32 integer conversion (one rounding) and
// scaled by 2^(e - 1075) through its exponent field. Operands whose pair
// parts would leave the normal float range take the hardware conversions.
__device__ __forceinline__ void emu_split_df(double v, float &hi, float &lo) {
    const uint64_t a = emu_bits(v);
    const uint32_t ah = (uint32_t)(a >> 32);
    const uint32_t e = (ah >> 20) & 0x7ffu;
    const uint64_t m = (a & kEmuFrac) | kEmuHidden;
    const uint32_t q = (uint32_t)(m >> 29), rem = (uint32_t)m & 0x1fffffffu;
    const uint32_t qh = q + ((rem > 0x10000000u || (rem == 0x10000000u && (q & 1u))) ? 1u : 0u);  // <= 2^24
    // exponent field e - 896 with the hidden bit of qh adding one (a carry to
    // 2^24 adds one more)
    const uint32_t hb = (ah & 0x80000000u) | (((e - 897u) << 23) + qh);
    const int32_t t = (int32_t)((uint32_t)m & 0x1fffffffu) - (int32_t)((qh - q) << 29);  // m - qh 2^29
    const float tf = __int2float_rn((ah & 0x80000000u) ? -t : t);
    const uint32_t lb = __float_as_uint(tf) + ((e - 1075u) << 23);  // tf 2^(e - 1075)
    bool ok = e - 950u < 200u;  // hi and lo (if not zero) normal floats
    hi = __uint_as_float(hb);
    lo = t == 0 ? 0.f : __uint_as_float(lb);
    if (!ok) {
        hi = __double2float_rn(v);
        lo = __double2float_rn(emu_native_sub(v, (double)hi));
    }
}

// RN(x + y) (SUB = false) or RN(x - y) (SUB = true). The smaller operand's
// significand is shifted right by the exponent difference with the lost bits
// jammed into bit 0; after the exact sum or difference, one more jammed right
// shift (which absorbs a carry out) and a left shift by the leading zeros
// bring the leading bit to 62, leaving 10 guard bits. A jammed bit always
// sits at or below bit 2 there, so it never decides a rounding on its own.
template <bool SUB>
__device__ __forceinline__ double emu_addsub(double x, double y) {
    const uint64_t a = emu_bits(x), b = emu_bits(y) ^ (SUB ? kEmuSign : 0ull);
    const bool sw = (a & ~kEmuSign) < (b & ~kEmuSign);  // order by magnitude
    const uint64_t big = sw ? b : a, small = sw ? a : b;
    const uint32_t gh = (uint32_t)(big >> 32), gl = (uint32_t)big;
    const uint32_t sh = (uint32_t)(small >> 32), sl = (uint32_t)small;
    const uint32_t ea = (gh >> 20) & 0x7ffu, eb = (sh >> 20) & 0x7ffu;
    const uint32_t d = ea - eb;  // >= 0 when both are normal
    // significands with the hidden bit at bit 62
    const uint64_t ma = ((uint64_t)((gh & 0xfffffu) | 0x100000u) << 42) | ((uint64_t)gl << 10);
    const uint64_t mb = ((uint64_t)((sh & 0xfffffu) | 0x100000u) << 42) | ((uint64_t)sl << 10);
    const uint32_t dc = d < 63u ? d : 63u;
    const uint64_t mt = mb >> dc;
    const uint64_t mbs = mt | ((mt << dc) != mb ? 1ull : 0ull);
    const bool same = ((gh ^ sh) & 0x80000000u) == 0u;
    const uint64_t s = same ? ma + mbs : ma - mbs;  // exact; >= 0 (big >= small)
    const uint64_t t0 = (s >> 1) | (s & 1ull);
    const int lz = __clzll((long long)t0) - 1;  // 0 .. 63
    const uint64_t t = t0 << lz;
    const int e = (int)ea + 1 - lz;  // biased exponent before rounding
    const uint32_t th = (uint32_t)(t >> 32), tl = (uint32_t)t;
    const uint32_t mhi = th >> 10, mlo = __funnelshift_r(tl, th, 10);
    const uint32_t rest = tl & 0x3ffu;
    const uint32_t up = (rest > 0x200u || (rest == 0x200u && (mlo & 1u))) ? 1u : 0u;
    const uint32_t rhi = (gh & 0x80000000u) | (((uint32_t)(e - 1) << 20) + mhi);
    uint64_t r = (((uint64_t)rhi << 32) | mlo) + up;
    const bool zero = s == 0ull;  // exact cancellation: +0
    r = zero ? 0ull : r;
    const bool bign = ea - 1u < 0x7feu;
    bool ok = bign && eb - 1u < 0x7feu && d < 64u && (zero || (uint32_t)(e - 1) < 2046u);
    if (bign && (small & ~kEmuSign) == 0ull) {  // big + 0 = big for a normal big
        r = big;
        ok = true;
    }
    if (!ok) r = emu_bits(SUB ? emu_native_sub(x, y) : emu_native_add(x, y));
    return emu_double(r);
}

// RN(sqrt(x)), x > 0 normal. V = the significand times 2^62 (times 2 for an
// odd exponent), in [2^62, 2^64). S0 = 24 bits of sqrt from the FP32
// reciprocal square root y0; two Newton corrections S += (V - S^2) y0 / 2
// bring the error to 2^-44 and 2^-66 relative, each residual exact in 64-bit
// modular arithmetic (it is far smaller than its operands) and read as a
// 32-bit window; so S2 = sqrt(V) 2^31 to within one unit of its 63 bits. The
// ten bits below the result's last decide the rounding unless they lie within
// that error of one half (1 in 256); then the exact sign of x - (midpoint)^2
// does (a square root is never a midpoint itself). Newton's iteration with a
// final exact remainder test, e.g. R. Brent and P. Zimmermann, "Modern
// Computer Arithmetic", 2010, section 1.5.1. 70 cycles in the probe (174 for
// the form before, which tested every result; 85 for this one testing always).
__device__ __forceinline__ double emu_sqrt_n(double x) {
    const uint32_t xh = emu_hi(x), xl = emu_lo(x);
    const uint32_t even = (xh >> 20) & 1u;  // biased exponent odd: the unbiased one is even
    const uint32_t a1 = emu_fsl(xl, xh, 11) | 0x80000000u, a0 = xl << 11;
    const uint32_t v1 = a1 >> even, v0 = __funnelshift_r(a0, a1, even);
    const float uf = __uint2float_rn(v1) * 0x1p-30f;  // V 2^-62 in [1, 4]
    const float y0 = emu_rsqrt_seed(uf);
    const uint32_t s0 = __float2uint_rn(uf * y0 * 0x1p23f);  // sqrt 2^23
    const uint64_t V = ((uint64_t)v1 << 32) | v0;
    // |V - s0^2 2^16| < 2^43
    const int64_t r0 = (int64_t)(V - (((uint64_t)s0 * s0) << 16));
    const int32_t c1 = __float2int_rn((float)(int32_t)(r0 >> 14) * y0 * 0x1p-3f);  // r0 y0 / 2 in units of 2^-46: * 2^-62 2^46 / 2
    const uint64_t S1 = ((uint64_t)s0 << 23) + (uint64_t)(int64_t)c1;  // sqrt 2^46
    const int64_t r1 = (int64_t)((V << 30) - S1 * S1);  // units of 2^-92, |r1| < 2^52
    const int32_t c2 = __float2int_rn((float)(int32_t)(r1 >> 22) * y0 * 0x1p-9f);  // r1 y0 / 2 in units of 2^-62
    const uint64_t S2 = (S1 << 16) + (uint64_t)(int64_t)c2;  // sqrt 2^62, within one unit
    uint64_t R = (S2 + 512ull) >> 10;  // [2^52, 2^53]
    if ((((uint32_t)S2 + 514u) & 1023u) < 4u) {
        R = (S2 + 510ull) >> 10;  // the candidate below the midpoint m / 2
        const uint64_t m = 2ull * R + 1ull;
        // sign of V 2^44 - m^2 (units of 2^-106), from the low 64 bits: |.| < 2^62
        if ((int64_t)((V << 44) - m * m) > 0) R += 1ull;
    }
    // exponent field of the result: (e - 1023 - odd) / 2 + 1023
    const uint32_t er = ((xh >> 20) + 1023u - (even ^ 1u)) >> 1;
    return emu_double(((uint64_t)(er - 1u) << 52) + R);
}

// RN(sqrt(x)), any x
__device__ __forceinline__ double emu_sqrt(double x) {
    const uint32_t e = emu_hi(x) >> 20;  // with the sign bit: > 2046 for negative x
    double r = emu_sqrt_n(x);
    if (!(e - 1u < 0x7feu)) r = emu_native_sqrt(x);
    return r;
}

// A divisor b prepared for several quotients: its significand mb and
// inv = 2^115 / mb to within one unit (inv in [2^62, 2^63]). FP32 seed v0 (24
// bits), two Newton corrections v += v (1 - b v) to 2^-44 and 2^-66 relative;
// each residual is small against 2^64, so its low 64 bits are all of it.
struct EmuDivisor {
    uint64_t mb, inv;
    uint32_t bh;  // high word of b: sign and exponent
};

__device__ __forceinline__ EmuDivisor emu_divisor(double b) {
    EmuDivisor D;
    const uint32_t bl = emu_lo(b);
    D.bh = emu_hi(b);
    const uint32_t b1 = (D.bh & 0xfffffu) | 0x100000u;
    D.mb = ((uint64_t)b1 << 32) | bl;
    const float bf = __uint_as_float((emu_fsl(bl, D.bh, 3) & 0x7fffffu) | 0x3f800000u);  // [1, 2), truncated
    const float rf = emu_rcp_seed(bf);
    const uint32_t v0 = __float2uint_rn(rf * 0x1p24f);  // 2^76 / mb, 2^23 .. 2^24
    // 2^76 - mb v0, |.| < 2^55
    const int64_t e0 = (int64_t)(0ull - ((uint64_t)bl * v0 + ((uint64_t)(b1 * v0) << 32)));
    const int32_t c1 = __float2int_rn((float)(int32_t)(e0 >> 25) * rf * 0x1p-4f);  // e0 v0 / 2^76 in units of 2^-23
    const uint64_t v1 = ((uint64_t)v0 << 23) + (uint64_t)(int64_t)c1;  // 2^99 / mb
    // 2^99 - mb v1, |.| < 2^57
    const int64_t e1 = (int64_t)(0ull - D.mb * v1);
    const int32_t c2 = __float2int_rn((float)(int32_t)(e1 >> 27) * rf * 0x1p-9f);
    D.inv = (v1 << 16) + (uint64_t)(int64_t)c2;  // 2^115 / mb
    return D;
}

// RN(x / y) with D = emu_divisor(y). X = ma inv is ma / mb 2^115 to within
// 2^53 (inv's unit times ma), so its leading 53 bits Q (a quotient >= 1: bits
// 63 on, else bits 62 on) are the quotient's floor, or one beside it when the
// quotient lies within 2^-9 units of a whole number; in every case the exact
// sign of x - (Q + 1/2) y, from the low 64 bits of ma 2^k - (2Q + 1) mb, says
// whether Q or Q + 1 is nearest (a quotient of two 53-bit significands is
// never a midpoint). Division by a scaled reciprocal with an exact remainder
// test, e.g. R. Brent and P. Zimmermann, "Modern Computer Arithmetic", 2010,
// 1.4.1. The test is taken always: rounding on the bits below Q and testing
// only the ambiguous ones took 80 cycles in a probe, this form 55.
__device__ __forceinline__ double emu_div_n(double x, const EmuDivisor &D) {
    const uint32_t xh = emu_hi(x), a0 = emu_lo(x);
    const uint32_t a1 = (xh & 0xfffffu) | 0x100000u;
    const uint32_t i1 = (uint32_t)(D.inv >> 32), i0 = (uint32_t)D.inv;
    const uint64_t m = (uint64_t)a0 * i1 + (uint64_t)a1 * i0 + (((uint64_t)a0 * i0) >> 32);  // < 2^64
    const uint64_t u = (uint64_t)a1 * i1 + (m >> 32);  // X >> 64, [2^50, 2^52)
    const uint32_t w1 = (uint32_t)m, w2 = (uint32_t)u, w3 = (uint32_t)(u >> 32);
    const uint32_t big = w3 >> 19, s = 2u - big;
    uint64_t Q = ((uint64_t)emu_fsl(w2, w3, s) << 32) | emu_fsl(w1, w2, s);
    // ma 2^(54 - big): its low word is zero
    const int64_t rem = (int64_t)(((uint64_t)(a0 << (22u - big)) << 32) - (2ull * Q + 1ull) * D.mb);
    Q += rem > 0 ? 1ull : 0ull;
    const uint32_t eh = (xh & 0xfff00000u) - (D.bh & 0xfff00000u) + ((1021u + big) << 20);
    return emu_double(((uint64_t)eh << 32) + Q);
}

// RN(x / 3), 3 a divisor prepared once: 2^115 / (3 2^51) = 2^64 / 3, rounded down
__device__ __forceinline__ double emu_div3_n(double x) {
    return emu_div_n(x, EmuDivisor{3ull << 51, 0x5555555555555555ull, 0x40080000u});
}

// RN(x / y): the unchecked quotient, or the hardware's when an operand lies
// outside [2^-500, 2^500)
__device__ __forceinline__ double emu_div(double x, const EmuDivisor &D, double y) {
    double r = emu_div_n(x, D);
    if (!(emu_within<500>(x) && emu_within<500>(y))) r = emu_native_div(x, y);
    return r;
}

__device__ __forceinline__ double emu_add(double x, double y) { return emu_addsub<false>(x, y); }
__device__ __forceinline__ double emu_sub(double x, double y) { return emu_addsub<true>(x, y); }

}  // namespace sphgpu
