// Reciprocals, reciprocal square roots and the limiter's harmonic half of
// FP64 numbers on the integer pipe.
//
// GB300 issues 2 FP64 operations per SM and cycle: a warp's FP64 add or
// multiply holds its scheduler's FP64 pipe for 70 to 82 cycles, a reciprocal
// refined there for 210, a reciprocal square root for 385.  The high half of a
// 64 x 64-bit product takes 18 cycles of the integer pipe, so a 62-bit
// fixed-point evaluation takes 75 to 150 cycles of a pipe that the FP64-bound
// kernels leave idle, and its result is rounded once, from 59 or more correct
// bits (the FP64 sequences round three to five times).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define MFG_HD __host__ __device__ __forceinline__
#else
#define MFG_HD inline
#endif

namespace mfg {

MFG_HD uint64_t umulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// High half of a product and of a square without the low partial product, whose
// place a constant takes: within 1 and 1.5 units of the exact value (the exact
// high half is within 1), in three and two 32-bit products instead of four.
MFG_HD uint32_t umulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
MFG_HD uint64_t mulhi_near(uint64_t a, uint64_t b) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return (uint64_t)ah * bh + ((uint64_t)umulhi32(ah, bl) + umulhi32(al, bh) + 1u);
}
MFG_HD uint64_t sqhi_near(uint64_t a) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
    return (uint64_t)ah * ah + (2 * (uint64_t)umulhi32(ah, al) + 1u);
}

MFG_HD int clz32(uint32_t x) {  // x != 0
#ifdef __CUDA_ARCH__
    return __clz((int)x);
#else
    return __builtin_clz(x);
#endif
}

MFG_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}

MFG_HD double double_of(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}

// High word of |x|: the order of magnitudes as integers.
MFG_HD int hi_abs(double x) { return (int)(bits_of(x) >> 32) & 0x7fffffff; }

// Bits of the float32 1/f, f in (1, 2), and 1/sqrt(f), f in (1, 4), relative
// error below 2^-22.
MFG_HD uint32_t rcp_seed_bits(uint32_t fbits) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
    return __float_as_uint(r);
#else
    float f;
    memcpy(&f, &fbits, 4);
    f = 1.0f / f;
    uint32_t b;
    memcpy(&b, &f, 4);
    return b;
#endif
}
MFG_HD uint32_t rsqrt_seed_bits(uint32_t fbits) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
    return __float_as_uint(r);
#else
    float f;
    memcpy(&f, &fbits, 4);
    f = 1.0f / __builtin_sqrtf(f);
    uint32_t b;
    memcpy(&b, &f, 4);
    return b;
#endif
}

MFG_HD int imin(int a, int b) { return a < b ? a : b; }
MFG_HD int imax(int a, int b) { return a > b ? a : b; }

// 2^126 / d for a normalised d (top bit set), relative error below 2^-59: the
// float32 seed r0 (e = 1 - x r0, |e| < 2^-21) corrected by r0 (1 + e + e^2).
MFG_HD uint64_t rcp_fixed(uint64_t d) {
    const uint32_t dh = (uint32_t)(d >> 32), dl = (uint32_t)d;
    uint32_t rb = rcp_seed_bits(0x3f800000u | ((dh & 0x7fffffffu) >> 8) | 1u);
    rb = rb < 0x3f000000u ? 0x3f000000u : rb > 0x3f7fffffu ? 0x3f7fffffu : rb;  // in [1/2, 1)
    const uint32_t R0 = ((rb & 0x7fffffu) | 0x800000u) << 7;                     // r0 2^31
    const uint64_t T = (uint64_t)dh * R0 + (((uint64_t)dl * R0) >> 32);          // (1 - e) 2^62
    const int64_t e = (int64_t)((1ull << 62) - T);
    const int32_t es = (int32_t)(e >> 18);
    const int64_t g = e + (((int64_t)es * es) >> 26);  // (e + e^2) 2^62
    const int32_t gh = (int32_t)(g >> 32);
    const uint32_t gl = (uint32_t)g;
    return ((uint64_t)R0 << 32) + (uint64_t)(((int64_t)gh * (int32_t)R0) << 2) + (((uint64_t)R0 * gl) >> 30);
}

constexpr uint64_t kMantMask = 0x000fffffffffffffull, kMantOne = 0x0010000000000000ull;

// Whether x is positive with an exponent away from the ends of the range (the
// integer forms below; everything else takes the FP64 sequences).
MFG_HD bool mid_positive(double x) {
    return (uint32_t)(bits_of(x) >> 32) - (40u << 20) < (1960u << 20);
}

// 1 / x for mid_positive(x).
MFG_HD double rcp_mid(double x) {
    const uint64_t b = bits_of(x);
    const uint64_t r = rcp_fixed(((b & kMantMask) | kMantOne) << 11);  // (2^62, 2^63]
    const uint32_t e = 2044u - (uint32_t)(b >> 52);
    return double_of(((uint64_t)e << 52) + ((r + 512) >> 10));  // r's top bit adds one to e
}

// 1 / sqrt(x) for mid_positive(x): x = m 2^(2h) with m in [1, 4), seed y0 =
// 1/sqrt(m) (1 + O(2^-21)), corrected by y0 (1 + e/2 + 3 e^2/8), e = 1 - m y0^2.
MFG_HD double rsqrt_mid(double x) {
    const uint64_t b = bits_of(x);
    const uint32_t ex = (uint32_t)(b >> 52);
    const uint32_t odd = (ex ^ 1u) & 1u;                                        // exponent ex - 1023 odd: m in [2, 4)
    const uint64_t m = ((b & kMantMask) | kMantOne) << (9 + odd);               // m 2^61
    const uint32_t mh = (uint32_t)(m >> 32), ml = (uint32_t)m;                  // m 2^29
    const uint32_t f = (0x3f800000u + (odd << 23)) | (uint32_t)((b >> 29) & 0x7fffffu) | 1u;
    uint32_t yb = rsqrt_seed_bits(f);                                           // 1/sqrt(m) in (1/2, 1)
    yb = yb < 0x3f000000u ? 0x3f000000u : yb > 0x3f7fffffu ? 0x3f7fffffu : yb;
    const uint32_t y0 = ((yb & 0x7fffffu) | 0x800000u) << 7;                    // y0 2^31
    const uint64_t p = (uint64_t)y0 * y0;                                       // y0^2 2^62, exact
    const uint32_t ph = (uint32_t)(p >> 32), pl = (uint32_t)p;
    // m y0^2 2^59 = m 2^61 * p 2^62 / 2^64
    const uint64_t q = (uint64_t)mh * ph + (((uint64_t)mh * pl) >> 32) + (((uint64_t)ml * ph) >> 32);
    const int64_t e = (int64_t)((1ull << 62) - (q << 3));                       // e 2^62
    const int32_t es = (int32_t)(e >> 18);
    const int64_t g = (e >> 1) + 3 * (((int64_t)es * es) >> 29);               // (e/2 + 3 e^2/8) 2^62
    const int32_t gh = (int32_t)(g >> 32);
    const uint32_t gl = (uint32_t)g;
    // y 2^63 in [2^62, 2^63]
    const uint64_t y =
        ((uint64_t)y0 << 32) + (uint64_t)(((int64_t)gh * (int32_t)y0) << 2) + (((uint64_t)y0 * gl) >> 30);
    const uint32_t h = (ex - 1023u - odd) >> 1;  // arithmetic halving of an even number, modulo 2^32
    const uint32_t e2 = 1021u - ((h & 0x40000000u) ? h | 0x80000000u : h);
    return double_of(((uint64_t)e2 << 52) + ((y + 512) >> 10));
}

// d1 d2 / (d1 + d2) for differences of the same sign, 0 otherwise: half the
// limited slope of the Tatsumi-Martinelli-Jameson limiter (compute_flux_3d.H:
// 33-65) in closed form, as the smaller difference times the larger one's
// share of the sum.  A non-finite difference gives NaN.
MFG_HD double limited_half(double d1, double d2) {
    const uint64_t b1 = bits_of(d1), b2 = bits_of(d2);
    const uint64_t a1 = b1 & 0x7fffffffffffffffull, a2 = b2 & 0x7fffffffffffffffull;
    const uint64_t hi = a1 > a2 ? a1 : a2, lo = a1 > a2 ? a2 : a1;
    const int eh = (int)(hi >> 52), el = (int)(lo >> 52);
    const uint64_t mh = ((hi & kMantMask) | kMantOne) << 10, ml = ((lo & kMantMask) | kMantOne) << 10;  // top bit 62
    uint64_t s = mh + (ml >> imin(eh - el, 63));
    const int k = (int)(~s >> 63);  // 1 when the sum stays below 2^63
    s <<= k;
    const uint64_t q = umulhi64(mh << k, rcp_fixed(s));  // share 2^62, in [2^61, 2^62]
    uint64_t r = umulhi64(ml << 1, q << 1);              // half 2^(...), in [2^61, 2^62 + 1]
    const int n = (int)((~r >> 62) & 1);
    r <<= n;
    uint64_t h = ((uint64_t)(uint32_t)(el - 1 - n) << 52) + ((r + 512) >> 10);
    h |= b1 & 0x8000000000000000ull;
    if ((int64_t)(b1 ^ b2) < 0 || el < 2) h = 0;
    if (eh == 0x7ff) h = 0x7ff8000000000000ull;
    return double_of(h);
}

// exp(-E/T) for E, T > 0 (the Arrhenius factor, E = Ea/RU), after the
// table-driven scheme of P. T. P. Tang (1989): with y = E log2(e) / T = n + j/64
// + r, exp(-E/T) = 2^-n 2^(-j/64) 2^-r, the last factor by its Taylor series
// (r < 2^-6: six terms leave 2^-58).  y has 59 correct bits, which the FP64
// form, a rounded product and a rounded quotient in front of the exponential,
// does not reach: its error is y 2^-53 and more.  About 300 cycles of the
// integer pipe against about 1900 of the FP64 pipe.
// E log2(e) as m 2^(e - 63), top bit of m set, comes from the host.
struct ExpScale {
    uint64_t m;
    int e;
};
inline ExpScale exp_scale(double num, double den) {  // host: E = num / den, both positive, finite, normal
    int xn, xd;
    const uint64_t n = (uint64_t)ldexp(frexp(num, &xn), 64), d = (uint64_t)ldexp(frexp(den, &xd), 53);
    const uint64_t log2e = 0xb8aa3b295c17f0bcull;  // 2^63 log2(e)
    const unsigned __int128 q = (unsigned __int128)n * log2e / d;
    int top = 127;
    while (!(uint64_t)(q >> top)) --top;
    return ExpScale{(uint64_t)(q >> (top - 63)), top + xn - xd - 74};
}

#define MFG_EXP2_TABLE /* 2^(-j/64) 2^63 */ \
    0x8000000000000000ull, 0x7e9f06067a4360baull, 0x7d41d96db915019dull, 0x7be86fb985689ddcull, \
    0x7a92be8a92436616ull, 0x7940bb9e2cffd89dull, 0x77f25ccdee6d7ae6ull, 0x76a7980f6cca15c2ull, \
    0x75606373ee921c97ull, 0x741cb5281e25ee34ull, 0x72dc8373be41a454ull, 0x719fc4b95f452d29ull, \
    0x70666f76154a7089ull, 0x6f307a412f074892ull, 0x6dfddbcbed791babull, 0x6cce8ae13c57ebdbull, \
    0x6ba27e656b4eb57aull, 0x6a79ad55e7f6fd10ull, 0x69540ec8f895722dull, 0x683199ed779592caull, \
    0x6712460a8fc24072ull, 0x65f60a7f79393e2eull, 0x64dcdec3371793d1ull, 0x63c6ba6455dcd8aeull, \
    0x62b39508aa836d6full, 0x61a3666d124bb204ull, 0x6096266533384a2bull, 0x5f8bccdb3d398841ull, \
    0x5e8451cfac061b5full, 0x5d7fad59099f22feull, 0x5c7dd7a3b17dcf75ull, 0x5b7ec8f19468bbc9ull, \
    0x5a827999fcef3242ull, 0x5988e20954889245ull, 0x5891fac0e95612c8ull, 0x579dbc56b48521baull, \
    0x56ac1f752150a563ull, 0x55bd1cdad49f699cull, 0x54d0ad5a753e077cull, 0x53e6c9da74b29ab5ull, \
    0x52ff6b54d8a89c75ull, 0x521a8ad704f3404full, 0x513821818624b40cull, 0x50582887dcb8a7e1ull, \
    0x4f7a993048d088d7ull, 0x4e9f6cd3967fdba8ull, 0x4dc69cdceaa72a9cull, 0x4cf022c9905bfd32ull, \
    0x4c1bf828c6dc54b8ull, 0x4b4a169b900c2d00ull, 0x4a7a77d47f7b84b1ull, 0x49ad159789f37496ull, \
    0x48e1e9b9d588e19bull, 0x4818ee218a3358eeull, 0x47521cc5a2e6a9e0ull, 0x468d6fadbf2dd4f3ull, \
    0x45cae0f1f545eb73ull, 0x450a6abaa4b77ecdull, 0x444c0740496d4294ull, 0x438fb0cb4f468808ull, \
    0x42d561b3e6243d8aull, 0x421d1461d66f2023ull, 0x4166c34c5615d0ecull, 0x40b268f9de0183baull,
#ifdef __CUDACC__
__device__ static const uint64_t kExp2Device[64] = {MFG_EXP2_TABLE};
#endif
#ifndef __CUDA_ARCH__
static const uint64_t kExp2Host[64] = {MFG_EXP2_TABLE};
#endif
MFG_HD uint64_t exp2_entry(int j) {
#ifdef __CUDA_ARCH__
    return __ldg((const unsigned long long*)kExp2Device + j);
#else
    return kExp2Host[j];
#endif
}

// T mid-range positive (mid_positive); false where the factor leaves the range
// of normal numbers.
MFG_HD bool exp_neg_over(const ExpScale& E, double T, double* out) {
    const uint64_t b = bits_of(T);
    const uint64_t rT = rcp_fixed(((b & kMantMask) | kMantOne) << 11);  // 2^126 / mantissa
    const uint64_t p = umulhi64(E.m, rT);                              // in [2^61, 2^63)
    const int s = 62 - E.e + ((int)(b >> 52) - 1023);                  // y = p 2^-s
    const uint64_t n = s < 64 ? p >> imax(s, 53) : 0;
    if (s < 53 || n > 1000) return false;                              // y >= 2^9 or 1001
    const uint64_t f = s <= 63 ? (p << (63 - s)) & 0x7fffffffffffffffull : s < 127 ? p >> (s - 63) : 0;  // 2^63 frac(y)
    const uint64_t z = umulhi64((f & 0x01ffffffffffffffull) << 1, 0xb17217f7d1cf79acull);  // r ln 2, 2^64
    uint64_t t = 0x002d82d82d82d82eull;  // 2^63 / 6!
    t = 0x0111111111111111ull - umulhi64(z, t);  // 2^63 / 5!
    t = 0x0555555555555555ull - umulhi64(z, t);  // 2^63 / 4!
    t = 0x1555555555555555ull - umulhi64(z, t);  // 2^63 / 3!
    t = 0x4000000000000000ull - umulhi64(z, t);  // 2^63 / 2!
    t = 0x8000000000000000ull - umulhi64(z, t);  // 2^63 / 1!
    t = 0x8000000000000000ull - umulhi64(z, t);
    const uint64_t w = umulhi64(exp2_entry((int)(f >> 57)), t);  // 2^-(j/64 + r) 2^62, in (2^61, 2^62]
    const int up = (int)(w >> 62);                        // 1 only for exactly 1
    const uint64_t m = w << (1 - up);                     // top bit at 62
    *out = double_of(((uint64_t)(uint32_t)(1023 - 1 - 1 + up - (int)n) << 52) + ((m + 512) >> 10));
    return true;
}

}  // namespace mfg
