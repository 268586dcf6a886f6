// FP64 products formed on the integer pipe, rounded exactly as the FP64
// multiply rounds them (IEEE 754 binary64, round to nearest even).
//
// On GB300 an FP64 warp instruction holds its SM sub-partition's FP64 pipe for
// 64 cycles, while integer instructions issue at up to one per cycle on
// another pipe.  The FP64 stencils are bound by the FP64 pipe, so a product
// that can be formed from the operand's bits with a handful of integer
// instructions frees FP64 time without changing a bit of the result:
//
//  * mul_pow2(x, f, k): x * f for f = 2^k.  For a normal x whose product is
//    normal, the product is exact and only adds k to the exponent field.
//  * mul6(x): x * 6.  The significand M (53 bits, leading one included) times
//    3 has 54 or 55 bits; it is shifted back to 53 bits and rounded to nearest,
//    ties to even, from the bits shifted out, and the exponent grows by the
//    shift plus one (the factor 2 of 6 = 2 * 3, exact).
//
// Zeros, subnormals, infinities, NaNs and products outside the normal range
// take the FP64 multiply itself (volatile inline PTX, so the compiler keeps
// that multiply inside its branch instead of computing it for every lane).
// The same functions compile for the host, where tests compare them with the
// host's multiply over random and edge-case operands.
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define SW_HD __host__ __device__ __forceinline__
#else
#define SW_HD inline
#endif

namespace sw {

SW_HD uint64_t f64_bits(double x) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    memcpy(&b, &x, sizeof b);
    return b;
#endif
}
SW_HD double f64_from_bits(uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, sizeof x);
    return x;
#endif
}
// The FP64 multiply, kept where it is written.
SW_HD double f64_mul_pipe(double a, double b) {
#if defined(__CUDA_ARCH__)
    double r;
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
#else
    volatile double va = a;
    return va * b;
#endif
}

// x * f with f = 2^k (|k| < 1023).
SW_HD double mul_pow2(double x, double f, int k) {
    const uint64_t b = f64_bits(x);
    const int e = (int)((b >> 52) & 0x7ff);
    if ((unsigned)(e - 1) < 2046u && (unsigned)(e + k - 1) < 2046u)
        return f64_from_bits(b + ((uint64_t)(int64_t)k << 52));
    return f64_mul_pipe(x, f);
}

// x * 6.
SW_HD double mul6(double x) {
    const uint64_t b = f64_bits(x);
    const int e = (int)((b >> 52) & 0x7ff);
    if ((unsigned)(e - 1) < 2043u) {  // normal x and a normal product: e + 3 <= 2046
        const uint64_t m = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;  // 53-bit significand
        const uint64_t p = m * 3u;                                               // 54 or 55 bits
        const int s = (p >> 54) ? 2 : 1;                                         // bits to drop
        uint64_t q = p >> s;
        const uint64_t rem = p & ((1ull << s) - 1), half = 1ull << (s - 1);
        q += (rem > half || (rem == half && (q & 1))) ? 1u : 0u;
        int ex = e + s;  // 3x's exponent ...
        if (q >> 53) {   // rounding carried into a 54th bit
            q >>= 1;
            ++ex;
        }
        ex += 1;  // ... times 2
        return f64_from_bits((b & 0x8000000000000000ull) | ((uint64_t)ex << 52) | (q & 0x000fffffffffffffull));
    }
    return f64_mul_pipe(x, 6.0);
}

// ---- general products, quotients and square roots on the integer pipe
//
// mul_int_fast(x, y, bad) = x * y, div_int_with(x, rcp_int(y), bad) = x / y
// and sqrt_int_fast(x, bad) = sqrt(x), each rounded once (to nearest, ties to
// even), for normal operands with a normal result (biased exponent at most
// 2045 before rounding); a division also takes a zero numerator.  For
// anything else -- other zeros, subnormals, infinities, NaNs, a result near or
// outside the ends of the normal range -- they set bad and the result is
// meaningless: the caller recomputes that value with the FP64 instruction.
// No FP64 instruction sits on their path, so none is issued: a predicated-off
// FP64 instruction still holds the FP64 pipe, and a fallback inside the
// product measured as slow as the multiply it replaces.
// mul_int holds that fallback (host checks); mul_any, div_any and sqrt_any
// call it.
SW_HD uint32_t f64_hi(double x) {
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2hiint(x);
#else
    return (uint32_t)(f64_bits(x) >> 32);
#endif
}
SW_HD uint32_t f64_lo(double x) {
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2loint(x);
#else
    return (uint32_t)f64_bits(x);
#endif
}
SW_HD double f64_of(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double((int)hi, (int)lo);
#else
    return f64_from_bits(((uint64_t)hi << 32) | lo);
#endif
}
SW_HD uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }  // one 32 x 32 -> 64 multiply-add
SW_HD uint32_t mulhi(uint32_t a, uint32_t b) { return (uint32_t)(wide(a, b) >> 32); }
// bits 32.. of (hi:lo) << s and the low word of (hi:lo) >> s, 0 <= s < 32
SW_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << s) >> 32);
#endif
}
SW_HD uint32_t shr_lo(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, s);
#else
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> s);
#endif
}
constexpr uint32_t kMantHi = 0x000fffffu, kHiddenHi = 0x00100000u, kSignExp = 0xfff00000u;

// Rounds the significand (mh:ml), 53 bits, on the 32 bits r below it (sticky:
// anything non-zero below r) to nearest even, and adds it to the word e that
// holds the sign and the exponent field less one.
SW_HD double round_pack(uint32_t e, uint32_t mh, uint32_t ml, uint32_t r, uint32_t sticky) {
    // r + (2^31 - 1) + (odd or sticky) carries exactly when the value is rounded up
    const uint32_t k = 0x7fffffffu + ((ml | (sticky < 1u ? sticky : 1u)) & 1u);
#if defined(__CUDA_ARCH__)
    uint32_t lo, hi;
    asm("{\n .reg .u32 t;\n add.cc.u32 t, %2, %3;\n addc.cc.u32 %0, %4, 0;\n addc.u32 %1, %5, %6;\n}"
        : "=r"(lo), "=r"(hi)
        : "r"(r), "r"(k), "r"(ml), "r"(mh), "r"(e));
    return f64_of(hi, lo);
#else
    const uint64_t c = ((uint64_t)r + k) >> 32;
    return f64_from_bits((((uint64_t)e << 32) + ((uint64_t)mh << 32)) + ml + c);
#endif
}

// The 106-bit product of the two significands in four 32-bit words p3..p0 (a
// 21-bit and a 32-bit half each: four multiply-adds, no shift before them);
// its leading one is bit 105 (top = 1) or 104, so the 53-bit result and the
// 32 bits below it are three funnel shifts by 20 + top.  In p0 a bit that r
// holds makes r odd, so p0 itself serves as the sticky word of a tie.
// The first form of this product (significands shifted to bit 63, 64-bit
// operations) took about half as many instructions again.  Heat FP64, two
// products per cell and bound by them (2^22 cells, tile 512): 1.29e11 ->
// 1.54e11 cell-updates/s; KS FP64 (2^20, tile 256) +0.8 %.
SW_HD double mul_int_fast(double x, double y, uint32_t &bad) {
    const uint32_t xh = f64_hi(x), yh = f64_hi(y), a0 = f64_lo(x), b0 = f64_lo(y);
    const uint32_t a1 = (xh & kMantHi) | kHiddenHi, b1 = (yh & kMantHi) | kHiddenHi;
    const uint64_t t0 = wide(a0, b0);
    const uint64_t t1 = wide(a1, b0) + (t0 >> 32);
    const uint64_t t2 = wide(a0, b1) + (uint32_t)t1;
    const uint64_t t3 = wide(a1, b1) + (t1 >> 32) + (t2 >> 32);
    const uint32_t p0 = (uint32_t)t0, p1 = (uint32_t)t2, p2 = (uint32_t)t3, p3 = (uint32_t)(t3 >> 32);
    const uint32_t top = p3 >> 9, s = top + 20u;
    const uint32_t mh = shr_lo(p2, p3, s), ml = shr_lo(p1, p2, s), r = shr_lo(p0, p1, s);
    const uint32_t ex = (xh >> 20) & 0x7ffu, ey = (yh >> 20) & 0x7ffu;
    // er = ex + ey - 1023 + top <= 2045: a rounding carry leaves the exponent field at most 2046
    bad |= (uint32_t)!(ex - 1u < 2046u && ey - 1u < 2046u && ex + ey + top - 1024u < 2045u);
    const uint32_t e = (xh & kSignExp) + (yh & kSignExp) + (top << 20) - (1024u << 20);
    return round_pack(e, mh, ml, r, p0);
}

// ---- quotients
//
// A correctly rounded FP64 quotient in software on the FP64 pipe is eight or
// more FP64 instructions (and a root as many) at 64 cycles or more of a
// sub-partition's pipe each; here it is about 60 integer ones.  Euler FP64
// swept (2^21 cells, tile 512; five to seven quotients and three roots per
// interface): 1.48e9 -> 2.80e9 cell-updates/s.
//
// The reciprocal of the divisor's significand b in [1, 2) to 2^-29, as a
// 32-bit fraction Y (Y / 2^32 <= 1 / b): the FP32 reciprocal approximation of
// b's leading 24 bits (error below 2^-22; any seed that close will do), then
// one Newton step y + y (1 - b y) in 32-bit integers.  bt holds b's leading 32
// bits (bit 31 set); the step takes bt + 1 for b and rounds down, so Y never
// exceeds the reciprocal.  Seed and step are the textbook ones; the quotient
// below corrects every remaining error exactly.
SW_HD float f32_rcp_seed(float x) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / x;
#endif
}
SW_HD float f32_rsqrt_seed(float x) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return (float)(1.0 / __builtin_sqrt((double)x));
#endif
}
SW_HD float f32_from_bits(uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float x;
    memcpy(&x, &b, sizeof x);
    return x;
#endif
}
// y in (0.5, 1) as y * 2^23: the significand bits of 1 + y
SW_HD uint32_t frac23(float y) {
    const float z = 1.0f + y;
#if defined(__CUDA_ARCH__)
    return __float_as_uint(z) - 0x3f800000u;
#else
    uint32_t b;
    memcpy(&b, &z, sizeof b);
    return b - 0x3f800000u;
#endif
}
SW_HD uint32_t rcp_newton(uint32_t bt, uint32_t y23) {
    const uint32_t yh = y23 << 8;                  // y * 2^31
    const uint64_t p = wide(bt, yh) + yh;          // (b + 2^-31) y * 2^62
    const int32_t e = (int32_t)~(uint32_t)(p >> 12);  // (1 - b y) * 2^50, rounded down
    const int32_t c = (int32_t)(((int64_t)(int32_t)yh * e) >> 32);
    return (yh << 1) + (uint32_t)(c >> 17);
}
struct RcpInt {
    uint32_t Y, n0, n1;  // the reciprocal; minus the significand (at bit 61) as two words
    uint32_t hi;         // the divisor's high word
};
SW_HD float rcp_int_arg(double b) {  // b's significand in [1, 2), 24 bits (never 1, so that y < 1)
    return f32_from_bits(0x3f800003u | (shl_hi(f64_lo(b), f64_hi(b), 3) & 0x007fffffu));
}
SW_HD RcpInt rcp_int_from(double b, float y) {
    const uint32_t bh = f64_hi(b), bl = f64_lo(b);
    const uint32_t bt = shl_hi(bl, bh, 11) | 0x80000000u;
    const uint64_t n = 0ull - ((((uint64_t)(bt >> 2)) << 32) | (bl << 9));
    return RcpInt{rcp_newton(bt, frac23(y)), (uint32_t)n, (uint32_t)(n >> 32), bh};
}
SW_HD RcpInt rcp_int(double b) { return rcp_int_from(b, f32_rcp_seed(rcp_int_arg(b))); }
// a / b from b's reciprocal: long division of the significands A, B (at bit
// 61) in two digits of 28 and 26 bits.  A digit is the remainder's leading 32
// bits times Y, at most 2.5 (first) and 1.44 (second) below the true quotient,
// so the remainders stay in [0, 2.5 B) -- below 2^64 -- and after the second
// digit one comparison makes Q = floor(A / B * 2^54) exact.  The quotient of
// two 53-bit significands is never halfway between two 53-bit numbers, so
// rounding needs no sticky bit.
SW_HD double div_int_with(double a, const RcpInt &b, uint32_t &bad) {
    const uint32_t ah = f64_hi(a), al = f64_lo(a);
    uint64_t R = ((uint64_t)((shl_hi(al, ah, 9) & 0x3fffffffu) | 0x20000000u) << 32) | (al << 9);
    const uint64_t n = ((uint64_t)b.n1 << 32) | b.n0;
    const uint32_t q1 = mulhi((uint32_t)(R >> 32), b.Y) >> 1;
    R = (R << 28) + wide(q1, b.n0) + ((uint64_t)(q1 * b.n1) << 32);
    const uint32_t q2 = mulhi((uint32_t)(R >> 32), b.Y) >> 3;
    R = (R << 26) + wide(q2, b.n0) + ((uint64_t)(q2 * b.n1) << 32);
    const uint64_t Q = wide(q1, 1u << 26) + q2 + (uint32_t)(R >= 0ull - n);
    const uint32_t top = (uint32_t)(Q >> 54);
    const uint64_t m = Q + top + 1u;
    const uint32_t ml = shr_lo((uint32_t)m, (uint32_t)(m >> 32), top + 1u), mh = (uint32_t)(m >> 32) >> (top + 1u);
    const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (b.hi >> 20) & 0x7ffu;
    const uint32_t sgn = (ah ^ b.hi) & 0x80000000u;
    const uint32_t e = (ea - eb + 1021u + top) << 20;
    const bool zero = ((ah << 1) | al) == 0;
    // er = ea - eb + 1022 + top in 1 .. 2045
    bad |= (uint32_t)!(eb - 1u < 2046u && (zero || (ea - 1u < 2046u && ea - eb + 1021u + top < 2045u)));
    return f64_of(zero ? sgn : ((e + mh) | sgn), zero ? 0u : ml);
}

// ---- square roots
//
// With m = x 4^-k in [1, 4) and M = m 2^62: a 32-bit root s1 of M from the
// FP32 reciprocal root y (biased down by 4 units of 2^-23, more than its error: s0 stays below the
// root and nothing overflows)
// and one correction by the remainder, s1 in (sqrt(M) - 2.1, sqrt(M) - 0.9];
// then one digit d of 23 bits more, the remainder times 1 / (2 s1) with y
// refined as a quotient's (s1 is the divisor).  s1 2^23 + d is S = floor(
// sqrt(m) 2^54) or S - 1, which the exact remainder decides.  A root of a
// 53-bit significand is never halfway between two 53-bit numbers either.
SW_HD double sqrt_int_from(double x, uint32_t &bad, float y) {
    const uint32_t xh = f64_hi(x), xl = f64_lo(x), ex = xh >> 20, odd = ex & 1u;  // odd: x's exponent is even
    const uint64_t n = ((uint64_t)(shl_hi(xl, xh, 11) | 0x80000000u) << 32) | (xl << 11);
    const uint64_t M = n >> odd;
    const uint32_t y23 = frac23(y) - 4u, y32 = y23 << 9;
    const uint32_t s0 = mulhi((uint32_t)(M >> 32), y32) << 1;
    const uint64_t r0 = M - wide(s0, s0);
    const uint32_t s1 = s0 + (mulhi((uint32_t)(r0 >> 14), y32) >> 18) - 1u;
    const uint64_t r1 = M - wide(s1, s1);
    const uint32_t Y = rcp_newton(s1 > 0x80000000u ? s1 : 0x80000000u, y23);
    const uint32_t d = (mulhi((uint32_t)(r1 >> 3), Y) - 4u) >> 6;
    // M 2^46 - (s1 2^23 + d)^2
    const uint64_t t = (r1 << 23) - (wide(s1, d) << 1);
    const uint64_t rem = (t << 23) - wide(d, d);
    const uint64_t S = wide(s1, 1u << 23) + d;
    const uint64_t m = (S + 2u + (uint32_t)(rem > (S << 1))) >> 2;
    bad |= (uint32_t)!(ex - 1u < 2046u);  // positive and normal
    const uint32_t e = (((ex + 1023u) >> 1) - 1u) << 20;
    return f64_of(e + (uint32_t)(m >> 32), (uint32_t)m);
}
SW_HD float sqrt_int_arg(double x) {  // x's significand in [1, 4), 24 bits
    const uint32_t xh = f64_hi(x), xl = f64_lo(x);
    return f32_from_bits((0x40000000u - (((xh >> 20) & 1u) << 23)) | (shl_hi(xl, xh, 3) & 0x007fffffu));
}
SW_HD double sqrt_int_fast(double x, uint32_t &bad) { return sqrt_int_from(x, bad, f32_rsqrt_seed(sqrt_int_arg(x))); }

SW_HD double mul_int(double x, double y) {
    uint32_t bad = 0;
    const double r = mul_int_fast(x, y, bad);
    return bad ? f64_mul_pipe(x, y) : r;
}

// ---- the same with the fallback at each operation, for Euler's long chains
//
// A cell-level flag and a second evaluation suit Heat and KS, whose cells leave
// the range together and rarely.  In an Euler run they do not: ahead of every
// front lies a band of cells whose momenta fall from 1e-16 to nothing, and each
// of them underflows in a product or two.  So each operation that meets such an
// operand calls the FP64 instruction itself.  The call keeps it out of line: a
// fallback that the compiler can turn into a predicated FP64 instruction costs
// as much as the FP64 operation would (8192 cells, tile 128: 11.0 ms for 256
// steps with one flag per interface, 8.9 ms on the FP64 pipe alone).
#if defined(__CUDACC__)
#define SW_SLOW static __host__ __device__ __noinline__
#else
#define SW_SLOW static
#endif
SW_SLOW double slow_mul(double x, double y) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(x, y);
#else
    return x * y;
#endif
}
SW_SLOW double slow_div(double x, double y) {
#if defined(__CUDA_ARCH__)
    return __ddiv_rn(x, y);
#else
    return x / y;
#endif
}
SW_SLOW double slow_sqrt(double x) {
#if defined(__CUDA_ARCH__)
    return __dsqrt_rn(x);
#else
    return __builtin_sqrt(x);
#endif
}
SW_SLOW double slow_half_min1(double r) {
    const double m = __builtin_fmin(r, 1.0);
#if defined(__CUDA_ARCH__)
    return __dmul_rn(0.5, m);
#else
    return 0.5 * m;
#endif
}
SW_HD double mul_any(double x, double y) {
    uint32_t bad = 0;
    double r = mul_int_fast(x, y, bad);
    if (bad) r = slow_mul(x, y);
    return r;
}
SW_HD double div_any(double a, double b, const RcpInt &ib) {
    uint32_t bad = 0;
    double r = div_int_with(a, ib, bad);
    if (bad) r = slow_div(a, b);
    return r;
}
SW_HD double sqrt_any(double x) {
    uint32_t bad = 0;
    double r = sqrt_int_fast(x, bad);
    if (bad) r = slow_sqrt(x);
    return r;
}
// x 2^k, k = -1 or 1 (f = 2^k)
SW_HD double pow2_any(double x, double f, int k) {
    const uint32_t hi = f64_hi(x);
    if (((hi >> 20) & 0x7ffu) - 2u < 2043u) return f64_of(hi + ((uint32_t)k << 20), f64_lo(x));
    return slow_mul(x, f);
}
// 0.5 min(r, 1), a NaN counting as 1 (fmin)
SW_HD double half_min1_any(double r) {
    const uint32_t hi = f64_hi(r);
    if ((int32_t)hi >= 0x3ff00000) return 0.5;  // 1 and above, infinity, NaN
    if (((hi >> 20) & 0x7ffu) - 2u < 2043u) return f64_of(hi - (1u << 20), f64_lo(r));
    return slow_half_min1(r);
}
// x == 0 and x < 0 without an FP64 comparison (which holds the FP64 pipe too)
SW_HD bool is_zero(double x) { return (f64_bits(x) << 1) == 0; }
SW_HD bool is_neg(double x) {
    const uint64_t b = f64_bits(x);
    return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull;
}

}  // namespace sw
