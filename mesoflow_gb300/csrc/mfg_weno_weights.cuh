// Nonlinear WENO5-JS weights (flux_schemes.H:373-446) in 64-bit fixed point.
//
// GB300 issues 2 FP64 operations per SM and cycle and 64 to 128 integer ones:
// a warp's FP64 add or multiply holds its scheduler's FP64 pipe for 82 cycles,
// a fused multiply-add for 70, while the high half of a 64 x 64-bit product
// takes 18 cycles of the integer pipe, which the order-5 flux kernels leave
// idle.  The weights are ratios of positive numbers, so they need no signs, no
// special values and no rounding modes, and fixed point gives them with errors
// of 2^-50 or less of their sum: indicators, squares, products, sums and
// reciprocals run here, beside the FP64 pipe that forms the differences and
// applies the weights.
//
// Such a weight is absolute: one of 1e-12, that of the stencil across a front,
// keeps 22 bits, and the corrections of the second-difference form are as large
// as the differences and cancel.  Where the stencil's differences are far above
// the values at the face the flux takes the weights in FP64 instead
// (weno_front, weno_front_edge).
//
// Everything is integer arithmetic but the 23-bit seed of the reciprocal, so
// every kernel that uses it gets the same bits.
#pragma once
#ifdef __CUDACC__
#include "mfg_common.cuh"
#else
#include "mfg_fixed.cuh"
#endif

namespace mfg {

// A cell difference split: |D| = m 2^(e - 1083), 2^60 <= m < 2^61 (zero and
// denormals read as about 2^-1023, far below the exponent floor).
struct WenoDiff {
    uint64_t m;
    int e;
    uint32_t sign;  // bit 31
};

MFG_HD WenoDiff weno_diff(uint64_t bits) {
    WenoDiff r;
    const uint32_t hi = (uint32_t)(bits >> 32);
    r.e = (int)((hi >> 20) & 0x7ffu);
    r.m = ((bits & 0x000fffffffffffffull) | 0x0010000000000000ull) << 8;
    r.sign = hi;
    return r;
}

// (eps + beta)^2 of a centre's three candidates up to one common factor:
// normalised 62 to 64-bit mantissas and the exponents of their square roots.
struct WenoInd {
    uint64_t dA, dB, dC;
    int eA, eB, eC;
};

// Exponent below which differences count as this one (2^-10: their squares are
// below eps = 1e-6), and 3 eps there in the units of the squares, 2^(2e - 2102).
constexpr int kWenoExpFloor = 1012;
constexpr uint64_t kWenoEps3 = 906694364710971881ull;  // 3e-6 * 2^78

// With D-, D+ the differences on both sides of the centre, 3 (eps + beta) is
// 3 eps + 4 D-^2 - 5 D- D+ + 4 D+^2 for the central candidate and, for the
// one-sided ones, that plus 6 D- (D- - D+) and 6 D+ (D+ - D-).  All three are
// at least 0.73 max(D-^2, D+^2), so the fixed point relative to the larger
// difference keeps them to 2^-50 at worst.
// RCP: also the reciprocals of the three 3 (eps + beta) as double bits (0 where
// they leave the exponent range), for the adjoint.
struct WenoIndR : WenoInd {
    uint64_t rA, rB, rC;
};

MFG_HD uint64_t ind_rcp_bits(uint64_t n, int z, int E) {
    const int e = 3061 - 2 * E + z;  // 3 (eps + beta) = n 2^(2E - 2102 - z), top bit of n set
    return e < 2 ? 0 : ((uint64_t)(uint32_t)(e - 1) << 52) + ((rcp_fixed(n) + 512) >> 10);
}

template <bool RCP>
MFG_HD WenoIndR weno_ind_full(const WenoDiff& a, const WenoDiff& b) {
    const int E = imax(imax(a.e, b.e), kWenoExpFloor);
    const uint64_t ma = a.m >> imin(E - a.e, 63), mb = b.m >> imin(E - b.e, 63);
    const uint64_t E1 = sqhi_near(ma), E2 = sqhi_near(mb);
    uint64_t X = mulhi_near(ma, mb);
    if ((a.sign ^ b.sign) >> 31) X = 0 - X;
    const uint64_t sC = ((E1 + E2) << 2) - 5 * X + (kWenoEps3 >> imin(2 * (E - kWenoExpFloor), 63));
    const uint64_t sA = sC + 6 * (E1 - X), sB = sC + 6 * (E2 - X);
    // each is at least 2^55: the high words are not zero
    const int zA = clz32((uint32_t)(sA >> 32)), zB = clz32((uint32_t)(sB >> 32)), zC = clz32((uint32_t)(sC >> 32));
    const uint64_t nA = sA << zA, nB = sB << zB, nC = sC << zC;
    WenoIndR r;
    r.dA = sqhi_near(nA);
    r.dB = sqhi_near(nB);
    r.dC = sqhi_near(nC);
    r.eA = 2 * E - zA;
    r.eB = 2 * E - zB;
    r.eC = 2 * E - zC;
    if (RCP) {
        r.rA = ind_rcp_bits(nA, zA, E);
        r.rB = ind_rcp_bits(nB, zB, E);
        r.rC = ind_rcp_bits(nC, zC, E);
    }
    return r;
}
MFG_HD WenoInd weno_ind(const WenoDiff& a, const WenoDiff& b) { return weno_ind_full<false>(a, b); }

// w 2^-62 2^k as the bits of a double, truncated (0 reads as 2^(k-62)).
MFG_HD uint64_t weight_bits(uint64_t w, int k) {
    uint32_t hi = (uint32_t)(w >> 32), lo = (uint32_t)w | 1u;
    int e = 1023 + 1 + k;
    if (hi == 0) {
        hi = lo;
        lo = 0;
        e -= 32;
    }
    const int z = clz32(hi);
    const uint64_t n = (((uint64_t)hi << 32) | lo) << z;  // top bit set: adds one to the exponent below
    return ((uint64_t)(uint32_t)(e - z - 1) << 52) + (n >> 11);
}

// A signed number of 2^-62 as the bits of a double.
MFG_HD uint64_t signed_weight_bits(int64_t v) {
    const uint64_t neg = (uint64_t)v >> 63;
    return weight_bits(neg ? 0 - (uint64_t)v : (uint64_t)v, 0) | (neg << 63);
}

// Weights of the two edges in cell m from the centres m-1 (dB), m (dC), m+1
// (dA).  With X = C A, Y = B A, Z = B C the left edge of face m+1 has the
// weights X, 6 Y, 3 Z over their sum for the far, middle and near candidate,
// the right edge of face m has Z, 6 Y, 3 X.  Returned: twice the far weight
// and the near weight of each edge, as double bits, and the near weights in
// units of 2^-62 (to be added before they are converted).
struct WenoWeights {
    uint64_t farL2, nearL, farR2, nearR;
    int64_t qL, qR;
};

MFG_HD WenoWeights weno_weights(uint64_t dB, int eB, uint64_t dC, int eC, uint64_t dA, int eA) {
    const int em = imin(imin(eA, eB), eC);
    // common exponent of the three products; four bits of headroom for the sums
    const uint64_t X = mulhi_near(dC, dA) >> imin(2 * (eB - em) + 4, 63);
    const uint64_t Y = mulhi_near(dB, dA) >> imin(2 * (eC - em) + 4, 63);
    const uint64_t Z = mulhi_near(dB, dC) >> imin(2 * (eA - em) + 4, 63);
    const uint64_t X3 = 3 * X, Z3 = 3 * Z, Y6 = 6 * Y;
    const uint64_t sL = X + Y6 + Z3, sR = Z + Y6 + X3;
    const int zL = clz32((uint32_t)(sL >> 32)), zR = clz32((uint32_t)(sR >> 32));
    // both reciprocals from that of the product: three products for one reciprocal
    const uint64_t nL = sL << zL, nR = sR << zR, P = mulhi_near(nL, nR);
    const int zP = (int)(~P >> 63);  // P in [2^62, 2^64)
    const uint64_t rP = rcp_fixed(P << zP), rL = mulhi_near(nR, rP) << zP, rR = mulhi_near(nL, rP) << zP;
    WenoWeights w;
    w.farL2 = weight_bits(mulhi_near(X << zL, rL), 1);
    w.qL = (int64_t)mulhi_near(Z3 << zL, rL);
    w.nearL = weight_bits((uint64_t)w.qL, 0);
    w.farR2 = weight_bits(mulhi_near(Z << zR, rR), 1);
    w.qR = (int64_t)mulhi_near(X3 << zR, rR);
    w.nearR = weight_bits((uint64_t)w.qR, 0);
    return w;
}

// Whether a face is beside a front: some difference of its stencil, of the state
// or of the Euler flux, large enough for the weights to depend on it (above the
// exponent floor) and far above the face's own values lam max(|u_L|, |u_R|) (with
// PRESSURE, the momentum along the sweep: and max(|f_L|, |f_R|), whose pressure
// that does not bound).  The fixed-point form's error is about 2^-54 of the
// differences, the FP64 candidates' 2^-51 of the values at the face: they meet
// near a ratio of 2^6.  Against 113-bit arithmetic, largest error over the face's
// values: a state of 1e-9 two faces from one of 1e3, 1e-6 in fixed point and 3e-16
// here; of 0.01 beside 1 (differences of 2^7), 2.6e-16 and 3.2e-16.
// topf, topu: the largest eB of the stencil's four centres: 3 (eps + beta) is 3 to
// 25 times the square of a difference (0.97 for the first one), so a difference's
// square counts to within 1.6 to 4.6 bits; the values' high words add as
// logarithms do, to within a bit.  A ratio between 2^6 and 2^8 is the first to
// count (2^9 where the first difference alone is large).  The line: over 60000
// random stencils of jumps from 2^-14 up and ratios from 1 up, faces kept on the
// fixed-point side are no further off than the candidates would be; one step higher
// some are, by 20%; one step lower, twice as many faces of a noisy field near zero
// take the candidates (64^3 right-hand side 608 -> 611 us).  Infinities, NaN and
// values above 2^880 count too.
constexpr int kFrontTop = 10, kFrontMost = 1900 << 20;
// Whether a stencil's differences (largest eB of its centres) are far above a value (high word of |v|).
MFG_HD bool front_above(int top, int value) {
    return top > imax((imin(value, kFrontMost) >> 19) + kFrontTop, 2 * kWenoExpFloor - 2);
}
MFG_HD bool weno_front(int topf, int topu, bool pressure, double fL, double fR, double uL, double uR, double lam) {
    const int l = hi_abs(lam) - 0x3ff00000;
    int mu = imin(imax(hi_abs(uL), hi_abs(uR)), kFrontMost), mf = (int)((unsigned)mu + (unsigned)l);
    if (pressure) {
        mf = imin(imax(mf, imax(hi_abs(fL), hi_abs(fR))), kFrontMost);
        mu = mf - l;
    }
    return front_above(topf, mf) || front_above(topu, mu);
}

// Six times one WENO5-JS edge of the cells a .. e, far upwind to far downwind
// (flux_schemes.H:373-446), as the mean of the candidates with positive FP64
// weights: its error is relative to the parts that make it up, whatever the
// cells beyond a front hold.  Explicit roundings: the sweep and the per-face
// form call it with the same cells and get the same bits.
struct Rn {
#ifdef __CUDA_ARCH__
    static MFG_HD double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
    static MFG_HD double mul(double a, double b) { return __dmul_rn(a, b); }
    static MFG_HD double add(double a, double b) { return __dadd_rn(a, b); }
    static MFG_HD double rcp(double x) { return rcp_pos(x); }
#else
    static MFG_HD double fma(double a, double b, double c) { return __builtin_fma(a, b, c); }
    static MFG_HD double mul(double a, double b) { return a * b; }
    static MFG_HD double add(double a, double b) { return a + b; }
    static MFG_HD double rcp(double x) { return 1.0 / x; }
#endif
};
// Weight of one candidate, not normalised: linear / (eps + 13/12 t^2 + q^2/4)^2.
MFG_HD double weno_front_weight(double t, double q, double linear) {
    const double s = Rn::fma(Rn::mul(0.25, q), q, Rn::fma(Rn::mul(13.0 / 12.0, t), t, 1e-6));
    const double r = Rn::rcp(s);
    return Rn::mul(linear, Rn::mul(r, r));
}
MFG_HD double weno_front_edge(double a, double b, double c, double d, double e) {
    const double w2 = weno_front_weight(Rn::add(Rn::fma(-2.0, b, a), c), Rn::fma(3.0, c, Rn::fma(-4.0, b, a)), 1.0);
    const double w1 = weno_front_weight(Rn::add(Rn::fma(-2.0, c, b), d), Rn::add(b, -d), 6.0);
    const double w0 = weno_front_weight(Rn::add(Rn::fma(-2.0, d, c), e), Rn::add(Rn::fma(3.0, c, Rn::mul(-4.0, d)), e), 3.0);
    const double v2 = Rn::fma(11.0, c, Rn::fma(-7.0, b, Rn::mul(2.0, a)));
    const double v1 = Rn::fma(2.0, d, Rn::fma(5.0, c, -b));
    const double v0 = Rn::fma(5.0, d, Rn::fma(2.0, c, -e));
    return Rn::mul(Rn::fma(w0, v0, Rn::fma(w1, v1, Rn::mul(w2, v2))), Rn::rcp(Rn::add(Rn::add(w2, w1), w0)));
}

// Weight of the first-order stencil (L, L, L, R, R, R) near the immersed
// boundary.  Its second differences are D and -D with D = R - L, both edges have
// the weight products X = c^2 b^2, Y = a^2 b^2, Z = a^2 c^2 of a = 3 eps, c = a +
// 4 D^2, b = a + 10 D^2, and the flux is (f_L + f_R)/2 - lam D W/2 with
//   W = (X + 2 Y - Z)/(X + 6 Y + 3 Z) = (1 + 2 u^2 - v^2)/(1 + 6 u^2 + 3 v^2),
// u = a/c, v = a/b, in [1/5, 1]: three reciprocals and eight products of the
// integer pipe, 2^-55 accurate, where the FP64 form took 25 operations beside the
// 19 of a regular face, in most warps near a boundary: fluxes of the 64^3
// catalyst step 3.65 -> 2.77 ms.
struct WenoCollapsed {
    uint64_t U, V;     // u, v: 2^62
    uint64_t den, rd;  // the denominator normalised (top bit 63), 2^126 over it
    int zd;            // its shift from units of 2^60
    uint64_t W;        // 2^62
};
MFG_HD WenoCollapsed weno_collapsed(const WenoDiff& d) {
    const int E = imax(d.e, kWenoExpFloor);
    const uint64_t m = d.m >> imin(E - d.e, 63), e2 = umulhi64(m, m), a = kWenoEps3 >> imin(2 * (E - kWenoExpFloor), 63);
    const uint64_t c = 4 * e2 + a, b = 10 * e2 + a;  // at least 2^57
    const int zc = clz32((uint32_t)(c >> 32)), zb = clz32((uint32_t)(b >> 32));
    WenoCollapsed r;
    r.U = umulhi64(a << zc, rcp_fixed(c << zc));
    r.V = umulhi64(a << zb, rcp_fixed(b << zb));
    const uint64_t one = 1ull << 60, u2 = umulhi64(r.U, r.U), v2 = umulhi64(r.V, r.V);
    const uint64_t num = one + 2 * u2 - v2, den = one + 6 * u2 + 3 * v2;  // den <= 10 2^60, num <= den
    r.zd = clz32((uint32_t)(den >> 32));
    r.den = den << r.zd;
    r.rd = rcp_fixed(r.den);
    r.W = umulhi64(num << r.zd, r.rd);
    return r;
}
// D dW/dD = -4 ((2 A - B) - W (6 A + 3 B))/den with A = u^2 (1 - u), B = v^2 (1 -
// v): the quotient without the factor, as double bits.
MFG_HD uint64_t weno_collapsed_slope(const WenoCollapsed& r) {
    const uint64_t one = 1ull << 62;
    const uint64_t A = umulhi64(umulhi64(r.U, r.U) << 2, one - r.U), B = umulhi64(umulhi64(r.V, r.V) << 2, one - r.V);  // 2^60
    const int64_t q = (int64_t)(2 * A) - (int64_t)B - (int64_t)(umulhi64(r.W, 6 * A + 3 * B) << 2);
    const uint64_t neg = (uint64_t)q >> 63;
    return weight_bits(umulhi64((neg ? 0 - (uint64_t)q : (uint64_t)q) << r.zd, r.rd), 0) | (neg << 63);
}

}  // namespace mfg
