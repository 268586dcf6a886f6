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

// ---- the general product on the integer pipe
//
// mul_int_fast(x, y, bad) = x * y, rounded once (to nearest, ties to even), for
// normal operands with a normal result (biased exponent at most 2045 before
// rounding).  For anything else -- zeros, subnormals, infinities, NaNs, a
// result near or outside the ends of the normal range -- it sets bad and the
// result is meaningless: the caller recomputes that value with the FP64
// multiply.  No FP64 instruction sits on its path, so none is issued: a
// predicated-off FP64 instruction still holds the FP64 pipe, and a fallback
// inside the product measured as slow as the multiply it replaces.
// mul_int holds that fallback (host checks).
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

SW_HD double mul_int(double x, double y) {
    uint32_t bad = 0;
    const double r = mul_int_fast(x, y, bad);
    return bad ? f64_mul_pipe(x, y) : r;
}

}  // namespace sw
