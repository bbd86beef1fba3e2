// Per-item bodies of the flow right-hand side (prim / face / flux / update),
// shared by the per-box launches (mfg_rhs.cu) and the batched persistent
// launches over all boxes of all levels (mfg_batch.cu).  See mfg_rhs.cu for
// the structure and the reference semantics.
#pragma once
#include "mfg_internal.h"
#include "mfg_physics.cuh"
#include "mfg_weno_weights.cuh"

namespace mfg {
namespace {

constexpr double kEpsWeno = 1e-6;

// FP64 sums and products as fused multiply-adds with 1 and -0 in registers:
// bitwise the add and the multiply, at the fused multiply-add's rate (a warp
// holds the FP64 pipe for 70 cycles; DADD and DMUL, and fused multiply-adds
// with an operand from the constant bank or an immediate, for 82).  The two
// constants pass through a shuffle so that they stay in registers; every lane
// of the warp constructs it.
struct Fp {
    double one, nz;
    __device__ __forceinline__ Fp() {
        one = __hiloint2double(__shfl_sync(0xffffffffu, 0x3ff00000, 0), 0);
        nz = __hiloint2double(__shfl_sync(0xffffffffu, (int)0x80000000, 0), 0);
    }
    // the constants as immediates, for code that part of a warp runs
    __device__ __forceinline__ explicit Fp(int) : one(1.0), nz(-0.0) {}
    __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return __fma_rn(b, -one, a); }
    __device__ __forceinline__ double mul(double a, double b) const { return __fma_rn(a, b, nz); }
};

// ---------------------------------------------------------------------------
// index helpers
// ---------------------------------------------------------------------------
struct Idx3 {
    int i, j, k;
};

__device__ __forceinline__ Idx3 delinear(int64_t t, const int lo[3], const int len[3]) {
    Idx3 r;
    split3(t, len[0], len[1], r.i, r.j, r.k);
    r.i += lo[0];
    r.j += lo[1];
    r.k += lo[2];
    return r;
}

// Euler flux of component c along d at one cell (consprim_funcs.H:48-81 with
// a unit normal e_d: the products with the zero normal components are exact
// zeros and drop out).  Rounding-faithful helpers keep the reference's
// separate multiply and add.
__device__ __forceinline__ double euler_flux(int c, int d, double u_c, double rho, double va, double vd,
                                             double p, double E) {
    if (c == RHO) return mul(rho, vd);
    if (c <= RHOW) {
        double t = mul(mul(rho, va), vd);
        return (c - 1 == d) ? add(t, p) : t;
    }
    if (c == RHOE) return mul(add(E, p), vd);
    return mul(u_c, vd);
}

// One WENO5-JS edge value (flux_schemes.H:373-446).  Inputs are the five
// stencil values ordered from the far upwind cell (a) to the far downwind
// cell (e); the right-biased edge passes them mirrored.  MIR selects the
// operand order of the reference's third candidate polynomial for the mirrored
// call.
template <bool MIR>
__device__ __forceinline__ double weno_edge(double a, double b, double c, double d, double e) {
    double t = (a - 2.0 * b) + c;
    double t2 = (a - 4.0 * b) + 3.0 * c;
    double b2 = (13.0 / 12.0) * (t * t) + 0.25 * (t2 * t2);
    t = (b - 2.0 * c) + d;
    double b1 = (13.0 / 12.0) * (t * t) + (0.25 * (b - d)) * (b - d);
    t = (c - 2.0 * d) + e;
    t2 = (3.0 * c - 4.0 * d) + e;
    double b0 = (13.0 / 12.0) * (t * t) + 0.25 * (t2 * t2);
    double v2 = MIR ? (11.0 * c - 7.0 * b) + 2.0 * a : (2.0 * a - 7.0 * b) + 11.0 * c;
    double v1 = (-b + 5.0 * c) + 2.0 * d;
    double v0 = (2.0 * c + 5.0 * d) - e;
    double a2 = 1.0 / ((kEpsWeno + b2) * (kEpsWeno + b2));
    double a1 = 6.0 * (1.0 / ((kEpsWeno + b1) * (kEpsWeno + b1)));
    double a0 = 3.0 * (1.0 / ((kEpsWeno + b0) * (kEpsWeno + b0)));
    double inv = 1.0 / ((a2 + a1) + a0);
    return ((1.0 / 6.0) * inv) * ((a2 * v2 + a1 * v1) + a0 * v0);
}

// Face value pair of the stencil s[0..5] = cells i-3 .. i+2 of face i:
// up = left-biased value (cells i-3..i+1), um = right-biased (cells i-2..i+2).
__device__ __forceinline__ void weno_face(const double s[6], double& up, double& um) {
    up = weno_edge<false>(s[0], s[1], s[2], s[3], s[4]);
    um = weno_edge<true>(s[5], s[4], s[3], s[2], s[1]);
}

// Sound speed sqrt(gamma p / rho), p = kap rho e (get_max_eigenvalue,
// flux_schemes.H:21-43).  Explicit roundings: equal states give equal speeds
// wherever it is compiled (the adjoint compares the two sides of a face).
__device__ __forceinline__ double eig_speed(double gam, double kap, double rhoe, double irho) {
    return sqrt_fast(__dmul_rn(__dmul_rn(gam, __dmul_rn(kap, rhoe)), irho));
}

// ---------------------------------------------------------------------------
// prim_kernel: per-cell scalars over grow(bx, 3)
// ---------------------------------------------------------------------------
template <int NS>
__device__ __forceinline__ void prim_body(const Fp& fp, const RhsBox& B, int64_t t) {
    int lo[3], len[3];
    for (int d = 0; d < 3; ++d) {
        lo[d] = B.lo[d] - MFG_NGROW;
        len[d] = B.hi[d] - B.lo[d] + 1 + 2 * MFG_NGROW;
    }
    const int64_t n = (int64_t)len[0] * len[1] * len[2];
    if (t >= n) return;
    const Idx3 c = delinear(t, lo, len);
    const Fab& S = B.sb;
    const int64_t o = S.off(c.i, c.j, c.k);
    const double rho = S.p[o + RHO * S.ns];
    const double m0 = S.p[o + RHOU * S.ns], m1 = S.p[o + RHOV * S.ns], m2 = S.p[o + RHOW * S.ns];
    const double E = S.p[o + RHOE * S.ns];
    double spec[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) spec[s] = (s < c_P.nspec) ? S.p[o + (NFLO + s) * S.ns] : 0.0;
    // cons_to_prim (consprim_funcs.H:9-23); one Newton-refined reciprocal of
    // the density replaces the reference's five divisions by it
    const double irho = rcp_pos(rho);
    const double vx = fp.mul(m0, irho), vy = fp.mul(m1, irho), vz = fp.mul(m2, irho);
    const double k2 = __fma_rn(vx, vx, __fma_rn(vy, vy, fp.mul(vz, vz)));
    const double rhoe = __fma_rn(-__dmul_rn(0.5, rho), k2, E);
    const double kap = thermo_kappa<NS>(rho, spec);
    const double pf = fp.mul(rhoe, kap);
    // get_max_eigenvalue's own-species terms (flux_schemes.H:21-43)
    const double mm = __fma_rn(m0, m0, __fma_rn(m1, m1, fp.mul(m2, m2)));
    const double reig = __fma_rn(-__dmul_rn(0.5, mm), irho, E);
    const double aown = eig_speed(1.0 + kap, kap, reig, irho);
    const Fab& X = B.aux;
    const int64_t q = X.off(c.i, c.j, c.k);
    X.p[q + AUX_VX * X.ns] = vx;
    X.p[q + AUX_VY * X.ns] = vy;
    X.p[q + AUX_VZ * X.ns] = vz;
    X.p[q + AUX_PF * X.ns] = pf;
    X.p[q + AUX_REIG * X.ns] = reig;
    X.p[q + AUX_AOWN * X.ns] = aown;
    X.p[q + AUX_KAP * X.ns] = kap;
}

// ---------------------------------------------------------------------------
// face_kernel: per-face scalars for direction d
// ---------------------------------------------------------------------------
// Faces of direction d (growHi(bx, d, 1)).
__device__ __forceinline__ int64_t face_count(const RhsBox& B, int d) {
    int64_t nf = 1;
    for (int e = 0; e < 3; ++e) nf *= B.hi[e] - B.lo[e] + 1 + (e == d);
    return nf;
}

// Whether face f of direction d takes the flux branch of face_body
// (Navier-Stokes terms on and face volume fraction >= 1/2), by the same
// arithmetic.
__device__ __forceinline__ bool face_active(const Fp& fp, const RhsBox& B, int d, const Idx3& f) {
    const Fab& S = B.sb;
    const int64_t sd = (d == 0) ? 1 : (d == 1) ? S.js : S.ks;
    const int64_t oR = S.off(f.i, f.j, f.k);
    const double* vf = S.p + VFRAC * S.ns;
    // 0.5 (a + b) >= 0.5 exactly when a + b >= 1 (the halving is exact)
    return c_P.do_ns && nonneg_ge(fp.add(vf[oR - sd], vf[oR]), 1.0);
}

// 1/x and 1/sqrt(x) of a positive x: fixed point on the integer pipe, or the
// FP64 forms at the ends of the exponent range.
__device__ __forceinline__ double face_rcp(double x) { return mid_positive(x) ? rcp_mid(x) : rcp_pos(x); }
__device__ __forceinline__ double face_rsqrt(double x) { return mid_positive(x) ? rsqrt_mid(x) : rsqrt(x); }

// Whether |v| < a for v and a^2, both of moderate size, by their exponents
// alone (true when |v| < 0.7 a; false when undecided).
__device__ __forceinline__ bool surely_below(double v, double a2) {
    const int ev = (__double2hiint(v) >> 20) & 0x7ff, ea = __double2hiint(a2) >> 20;
    return ea > 0 && 2 * (ev + 1 - 1023) < ea - 1023;  // |v|^2 < 2^(2 (ev + 1)) <= 2^ea <= a^2
}

// The two sides' shares of an AUSM+-up face (flux_schemes.H:107-181, beta =
// 1/8) at the Mach number M, sign = +1 for the left side and -1 for the right; q
// = M^2 - 1, and the |M| <= 1 tests run on the integer pipe.  Four times the
// pressure split: (M + sign)^2 (2 - sign M) + 4 sign alpha M (M^2 - 1)^2 below
// |M| = 1, as g and M q^2, and exactly 4 or 0 above.
__device__ __forceinline__ void ausm_split(const Fp& fp, double M, double sign, double q, double& g, double& mq2) {
    const double a = __fma_rn(sign, fp.one, M);
    const bool sub = abs_le(M, 1.0), on = sign > 0.0 ? is_positive(M) : is_negative(M);
    g = sub ? fp.mul(fp.mul(a, a), __fma_rn(-sign, M, 2.0)) : (on ? 4.0 : 0.0);
    mq2 = sub ? fp.mul(M, fp.mul(q, q)) : 0.0;
}
// Four times one side's Mach split: sign ((M + sign)^2 + (M^2 - 1)^2/2) below
// |M| = 1, 4 M or 0 above (without the sign).
__device__ __forceinline__ double ausm_mach4(const Fp& fp, double M, double sign, double q) {
    const double a = __fma_rn(sign, fp.one, M);
    const bool on = sign > 0.0 ? is_positive(M) : is_negative(M);
    return abs_le(M, 1.0) ? __fma_rn(0.5, fp.mul(q, q), fp.mul(a, a)) : (on ? __dmul_rn(4.0 * sign, M) : 0.0);
}

// Face f of direction d.  SOLID_SIDE: the caller knows the face is not
// active and the pass is the split form of orders 1/2 with Navier-Stokes
// terms (face_split_kernel); the flux branch and the first-order fallback
// test (used only by the flux branch and the stored face scalars of orders
// 4/5) are compiled out, the remaining arithmetic is the same.  ACTIVE: the
// caller knows that it is active.
//
// FP64 issue bounds the flux branch of orders 1/2.  Its reciprocals, square
// roots and limiters run in fixed point on the integer pipe (mfg_fixed.cuh),
// its sums and products as register-operand multiply-adds (Fp), and every
// rounding is explicit, so the one-pass and the listed form agree bitwise.
// About 150 FP64 operations per face of one species at 70 cycles (205 at 82
// with the refined reciprocals there): face passes of a 256^3 sphere-pack step
// 50.4 -> 38.0 ms, and 36.8 with the factors of four of the splits, the viscosity
// and the conductivity inside multiply-adds; the listed form keeps the FP64 pipe
// 83% busy.
//
// HIGH: orders 4 and 5, else 1 and 2 (the caller has the order from the host,
// so each kernel holds the registers of its own branch).
template <int NS, bool HIGH, bool SOLID_SIDE = false, bool ACTIVE = false>
__device__ __forceinline__ void face_body_at(const Fp& fp, const RhsBox& B, int d, const Idx3& f) {
    const DevParams& P = c_P;
    const Fab& S = B.sb;
    const int64_t sd = (d == 0) ? 1 : (d == 1) ? S.js : S.ks;
    const int t1 = (d + 1) % 3, t2 = (d + 2) % 3;
    const int64_t st1 = (t1 == 0) ? 1 : (t1 == 1) ? S.js : S.ks;
    const int64_t st2 = (t2 == 0) ? 1 : (t2 == 1) ? S.js : S.ks;
    const int64_t oR = S.off(f.i, f.j, f.k);  // right cell: face i separates i-1 and i
    const int64_t oL = oR - sd;
    const double* vf = S.p + VFRAC * S.ns;
    const int ord = P.order_hyp;

    bool fallback = false;
    if (!SOLID_SIDE) {
#pragma unroll
        for (int q = -3; q <= 2; ++q) fallback |= below_one(vf[oR + q * sd]);
    }
    // face volume fraction 0.5 (a + b) >= 0.5, i.e. a + b >= 1 (the halving is exact)
    const bool active = ACTIVE || (!SOLID_SIDE && P.do_ns && nonneg_ge(fp.add(vf[oL], vf[oR]), 1.0));

    double lam = 0.0;                        // orders 4, 5: LLF eigenvalue
    double uL[NCONS + NS], uR[NCONS + NS];   // orders 1, 2: advected face states, E + p for the energy
    double wL = 0.0, wR = 0.0, ph4 = 0.0;    // orders 1, 2: mass-flux weights, four times the interface pressure
    double vis[3] = {0.0, 0.0, 0.0}, vise2 = 0.0;  // viscous stresses over mu; twice the viscous work over mu
    double mu = 0.0, kc = 0.0, therm = 0.0;  // viscosity, conductivity; heat conduction over k

    if (active) {
        if (HIGH) {
            const Fab& X = B.aux;
            const int64_t qL = X.off(f.i, f.j, f.k) - ((d == 0) ? 1 : (d == 1) ? X.js : X.ks);
            const int64_t qR = X.off(f.i, f.j, f.k);
            const double* vd = X.p + (AUX_VX + d) * X.ns;
            const double veln = max_nonneg(fabs(vd[qL]), fabs(vd[qR]));
            const double aL = X.p[qL + AUX_AOWN * X.ns];
            double aR;
            if (ord == 5) {
                // presR is evaluated with the left cell's species (flux_schemes.H:33):
                // kappa of the left cell, but for the background-gas family, whose
                // kappa depends on the density too
                const double rhoR = S.p[oR + RHO * S.ns];
                double kapL = X.p[qL + AUX_KAP * X.ns];
                if (P.thermo_kind == MFG_THERMO_BG_GAS) {
                    double specL[NS];
#pragma unroll
                    for (int s = 0; s < NS; ++s) specL[s] = (s < P.nspec) ? S.p[oL + (NFLO + s) * S.ns] : 0.0;
                    kapL = thermo_kappa<NS>(rhoR, specL);
                }
                aR = eig_speed(1.0 + X.p[qR + AUX_KAP * X.ns], kapL, X.p[qR + AUX_REIG * X.ns], rcp_pos(rhoR));
            } else {
                aR = X.p[qR + AUX_AOWN * X.ns];
            }
            lam = fp.add(max_nonneg(aL, aR), veln);
        } else {
            // AUSM+-up (flux_schemes.H:185-310) on first- or second-order states
            // (MUSCL: u_L + h and u_R - h with h the limited half slope)
            const int nc = NCONS + P.nspec;
#pragma unroll
            for (int c = 0; c < NCONS + NS; ++c) {
                if (c >= nc) { uL[c] = uR[c] = 0.0; continue; }
                const double* u = S.p + ((c < NCONS) ? c : c + (NFLO - NCONS)) * S.ns;
                uL[c] = u[oL];
                uR[c] = u[oR];
                if (ord == 2 && !fallback) {
                    const double h = limited_half(fp.sub(u[oR + sd], uR[c]), fp.sub(uL[c], u[oL - sd]));
                    uL[c] = fp.add(uL[c], h);
                    uR[c] = fp.sub(uR[c], h);
                }
            }
            const double rL = uL[RHO], rR = uR[RHO];
            const double irL = face_rcp(rL), irR = face_rcp(rR);
            // internal energy rho e = E - |m|^2 / (2 rho) from the momenta
            const double k2L = fp.mul(
                __fma_rn(uL[RHOU], uL[RHOU], __fma_rn(uL[RHOV], uL[RHOV], fp.mul(uL[RHOW], uL[RHOW]))), irL);
            const double k2R = fp.mul(
                __fma_rn(uR[RHOU], uR[RHOU], __fma_rn(uR[RHOV], uR[RHOV], fp.mul(uR[RHOW], uR[RHOW]))), irR);
            // kappa = gamma - 1 of both states as one division each, or as its
            // numerator and denominator: 2 (gamma - 1)/(gamma + 1) = n/(d + n/2),
            // with reciprocals of the integer pipe
            double kL = P.gm1_single, kR = P.gm1_single, afL = P.astar_fac, afR = P.astar_fac;
            if (P.thermo_kind != MFG_THERMO_MASS_SINGLE) {
                double n, dn;
                thermo_ratio<NS>(rL, uL + NCONS, n, dn);
                kL = fp.mul(n, face_rcp(dn));
                afL = fp.mul(n, face_rcp(__fma_rn(0.5, n, dn)));
                thermo_ratio<NS>(rR, uR + NCONS, n, dn);
                kR = fp.mul(n, face_rcp(dn));
                afR = fp.mul(n, face_rcp(__fma_rn(0.5, n, dn)));
            }
            const double pL = fp.mul(__fma_rn(-0.5, k2L, uL[RHOE]), kL), pR = fp.mul(__fma_rn(-0.5, k2R, uR[RHOE]), kR);
            const double vL = fp.mul((d == 0) ? uL[RHOU] : (d == 1) ? uL[RHOV] : uL[RHOW], irL);
            const double vR = fp.mul((d == 0) ? uR[RHOU] : (d == 1) ? uR[RHOV] : uR[RHOW], irR);
            // E + p: what the energy flux advects, and rho times the total enthalpy
            // gamma/(gamma-1) p/rho + |v|^2/2
            uL[RHOE] = fp.add(uL[RHOE], pL);
            uR[RHOE] = fp.add(uR[RHOE], pR);
            const double rsum = fp.add(rL, rR);
            // a_hat = a*^2 / max(a*, |v|) per side, a_1/2 = min(a_hat_L, a_hat_R)
            // and its reciprocal.  On a subsonic side (a* >= |v|) a_hat = a*, so
            // when both sides are subsonic a_1/2 is the square root of the smaller
            // a*^2: a_1/2 = m rsqrt(m) and 1/a_1/2 = rsqrt(m).  Otherwise each
            // side as a* or a*^2/|v| (and |v|/a*^2), the smaller.
            const double as2L = fp.mul(afL, fp.mul(uL[RHOE], irL)), as2R = fp.mul(afR, fp.mul(uR[RHOE], irR));
            double ah, iah;
            if ((surely_below(vL, as2L) || nonneg_ge(as2L, fp.mul(vL, vL))) &&
                (surely_below(vR, as2R) || nonneg_ge(as2R, fp.mul(vR, vR)))) {
                const double m = min_nonneg(as2L, as2R);
                iah = face_rsqrt(m);
                ah = fp.mul(m, iah);
            } else {
                double irs = face_rsqrt(as2L);
                double ahL = fp.mul(as2L, irs), iahL = irs;
                if (!nonneg_ge(ahL, fabs(vL))) {
                    ahL = fp.mul(as2L, rcp_pos(fabs(vL)));
                    iahL = fp.mul(fabs(vL), rcp_pos(as2L));
                }
                irs = face_rsqrt(as2R);
                double ahR = fp.mul(as2R, irs), iahR = irs;
                if (!nonneg_ge(ahR, fabs(vR))) {
                    ahR = fp.mul(as2R, rcp_pos(fabs(vR)));
                    iahR = fp.mul(fabs(vR), rcp_pos(as2R));
                }
                const bool left = nonneg_le(ahL, ahR);
                ah = left ? ahL : ahR;
                iah = left ? iahL : iahR;
            }
            const double ML = fp.mul(vL, iah), MR = fp.mul(vR, iah);
            const double qL = __fma_rn(ML, ML, -fp.one), qR = __fma_rn(MR, MR, -fp.one);
            // mean Mach number Mb^2 = (ML^2 + MR^2)/2 = 1 + (qL + qR)/2
            const double qs = fp.add(qL, qR), Mb2 = __fma_rn(0.5, qs, 1.0);
            // the splits, and four times M_1/2: with both sides subsonic the Mach splits'
            // sum in closed form, (ML + MR) (2 + (ML - MR) Mb^2), which does not cancel at
            // low Mach numbers as the difference of two terms near one does.  Below
            // 1/2 the pressure splits' g as 2 +- M (3 - M^2): one rounding of its size
            // instead of the product's four (momentum of an order-2 right-hand side
            // 15% closer to extended precision) in half the operations (face passes of
            // a 256^3 sphere-pack step 36.8 -> 35.7 ms); beyond, the product, which
            // keeps its digits where g goes to zero.
            double gL, gR, mqL, mqR, mm4;
            if (imax(hi_abs(ML), hi_abs(MR)) < 0x3fe00000) {
                gL = __fma_rn(ML, __fma_rn(-ML, ML, 3.0), 2.0);
                gR = __fma_rn(-MR, __fma_rn(-MR, MR, 3.0), 2.0);
                mqL = fp.mul(ML, fp.mul(qL, qL));
                mqR = fp.mul(MR, fp.mul(qR, qR));
                mm4 = fp.mul(fp.add(ML, MR), __fma_rn(fp.sub(ML, MR), Mb2, 2.0));
            } else {
                ausm_split(fp, ML, 1.0, qL, gL, mqL);
                ausm_split(fp, MR, -1.0, qR, gR, mqR);
                if (abs_le(ML, 1.0) && abs_le(MR, 1.0))
                    mm4 = fp.mul(fp.add(ML, MR), __fma_rn(fp.sub(ML, MR), Mb2, 2.0));
                else
                    mm4 = fp.sub(ausm_mach4(fp, ML, 1.0, qL), ausm_mach4(fp, MR, -1.0, qR));
            }
            // M_o = sqrt(min(1, max(Mb^2, 0.3^2))) as x rsqrt(x) on the clamped x
            const double xmo = min_nonneg(1.0, max_nonneg(pos_part(Mb2), 0.3 * 0.3));
            const double Mo = fp.mul(xmo, face_rsqrt(xmo));
            const double fa = fp.mul(Mo, __fma_rn(-Mo, fp.one, 2.0));
            const double fr = fp.mul(fa, rsum);
            // pressure diffusion: M_1/2 less (1 - Mb^2)^+ (p_R - p_L) / (4 fa rho_1/2
            // a_1/2^2) with rho_1/2 = (rho_L + rho_R)/2, as 4 M_1/2 less
            // (-qs)^+ (p_R - p_L) / (fa (rho_L + rho_R) a_1/2^2)
            const double pd = fp.mul(fp.mul(pos_part(-qs), fp.sub(pR, pL)), fp.mul(iah, iah));
            // M_1/2, its modulus with the parabola below 0.3, and the pressure
            // splits, each times four (exact scales, taken back where they cost nothing)
            const double M4 = __fma_rn(-pd, face_rcp(fr), mm4);
            double mod4 = fabs(M4);
            if (nonneg_le(mod4, 4.0 * 0.3)) mod4 = __dmul_rn(__fma_rn(M4, M4, 16.0 * (0.3 * 0.3)), 0.25 * (1.0 / (2.0 * 0.3)));
            // alpha = 3/16 (-4 + 5 fa^2) as (15/16 fa) fa - 3/4
            const double a4 = __fma_rn(__dmul_rn(15.0 / 4.0, fa), fa, -3.0);
            const double PL4 = __fma_rn(a4, mqL, gL), PR4 = __fma_rn(-a4, mqR, gR);
            const double pu16 = fp.mul(fp.mul(fp.mul(PL4, PR4), fp.mul(fr, ah)), fp.sub(vR, vL));
            ph4 = __fma_rn(-3.0 / 16.0, pu16, __fma_rn(PL4, pL, fp.mul(PR4, pR)));
            // mass-flux weights with the wave speed folded in: the flux of a
            // component (M/2 (fL + fR) - |M|/2 (fR - fL)) a_half is wL fL + wR fR
            // with wL = (M + |M|) a_half / 2, wR = (M - |M|) a_half / 2
            const double ah8 = __dmul_rn(0.125, ah);
            const double cmh = fp.mul(M4, ah8), cmod = fp.mul(mod4, ah8);
            wL = fp.add(cmh, cmod);
            wR = fp.sub(cmh, cmod);
        }
        // Viscous stress (compute_flux_3d.H:293-367), lagged primitive
        // velocities.  Only the row of the face normal is needed: off the diagonal
        // mu (dV_a/dx_d + dV_d/dx_a), on it mu (2 dV_d/dx_d - 2/3 div V), where
        // the divergence needs the two transverse diagonal derivatives, so
        // mu (4/3 dV_d/dx_d - 2/3 (dV_t1/dx_t1 + dV_t2/dx_t2)): 7 of the 9
        // gradients.  A transverse derivative is ((a + b) - (c + d)) / (4 dx);
        // all scales sit in multiply-adds.
        const double* V0 = S.p + VELX * S.ns;
        const double* V1 = S.p + VELY * S.ns;
        const double* V2 = S.p + VELZ * S.ns;
        const double* Vd = (d == 0) ? V0 : (d == 1) ? V1 : V2;
        const double* Vt1 = (t1 == 0) ? V0 : (t1 == 1) ? V1 : V2;
        const double* Vt2 = (t2 == 0) ? V0 : (t2 == 1) ? V1 : V2;
        const double vdL = Vd[oL], vdR = Vd[oR], v1L = Vt1[oL], v1R = Vt1[oR], v2L = Vt2[oL], v2R = Vt2[oR];
        const double e1 = fp.sub(fp.add(Vd[oL + st1], Vd[oR + st1]), fp.add(Vd[oL - st1], Vd[oR - st1]));
        const double e2 = fp.sub(fp.add(Vd[oL + st2], Vd[oR + st2]), fp.add(Vd[oL - st2], Vd[oR - st2]));
        const double s1 = fp.sub(fp.add(Vt1[oL + st1], Vt1[oR + st1]), fp.add(Vt1[oL - st1], Vt1[oR - st1]));
        const double s2 = fp.sub(fp.add(Vt2[oL + st2], Vt2[oR + st2]), fp.add(Vt2[oL - st2], Vt2[oR - st2]));
        // viscosity always from cells (i,j,k) and (i-1,j,k) (compute_flux_3d.H:179)
        mu = (P.visc_mode == MFG_TRANSPORT_CONST)
                 ? P.visc_hm
                 : harmonic_mean(blend(P.visc_mode, P.visc_gas, P.visc_solid, vf[oR]),
                                 blend(P.visc_mode, P.visc_gas, P.visc_solid, vf[oR - 1]));
        const double taud = __fma_rn(fp.sub(vdR, vdL), B.i43[d], __fma_rn(s1, B.iq23[t1], fp.mul(s2, B.iq23[t2])));
        const double tau1 = __fma_rn(fp.sub(v1R, v1L), B.idx[d], fp.mul(e1, B.iq[t1]));
        const double tau2 = __fma_rn(fp.sub(v2R, v2L), B.idx[d], fp.mul(e2, B.iq[t2]));
        // over mu, which the flux takes in its multiply-adds; twice the viscous
        // work sum_a tau_{d a} v_a of the energy flux
        vise2 = __fma_rn(taud, fp.add(vdL, vdR), __fma_rn(tau1, fp.add(v1L, v1R), fp.mul(tau2, fp.add(v2L, v2R))));
#pragma unroll
        for (int a = 0; a < 3; ++a) vis[a] = (a == d) ? taud : (a == t1) ? tau1 : tau2;
    }
    if (P.do_ns) {
        // heat conduction (compute_flux_3d.H:373-374), conductivity from (i,j,k),(i-1,j,k)
        kc = (P.cond_mode == MFG_TRANSPORT_CONST)
                 ? P.cond_hm
                 : harmonic_mean(blend(P.cond_mode, P.cond_gas, P.cond_solid, vf[oR]),
                                 blend(P.cond_mode, P.cond_gas, P.cond_solid, vf[oR - 1]));
        const double* T = S.p + TEMP * S.ns;
        therm = fp.mul(fp.sub(T[oR], T[oL]), B.idx[d]);
    }
    if (!HIGH && (SOLID_SIDE || P.do_ns)) {
        // AUSM+-up: the face thread holds the face states and the scheme scalars,
        // so it writes every component's complete flux (no per-component pass).
        const Fab& O = B.flx[d];
        const int64_t qo = O.off(f.i, f.j, f.k);
        const Fab& U = B.uflux[d];
        const int64_t qu = U.p ? U.off(f.i, f.j, f.k) : 0;
#pragma unroll
        for (int c = 0; c < NCONS + NS; ++c) {
            if (c >= NCONS + P.nspec) break;
            const int sc = (c < NCONS) ? c : c + (NFLO - NCONS);
            double F = 0.0;
            if (active) {
                F = __fma_rn(wR, uR[c], fp.mul(wL, uL[c]));
                if (c == 1 + d) F = __fma_rn(0.25, ph4, F);
                if (c >= NCONS && !is_one(P.advect_flag[c - NCONS])) F = fp.mul(P.advect_flag[c - NCONS], F);
                if (c >= RHOU && c <= RHOW) F = __fma_rn(-mu, vis[c - 1], F);
                if (c == RHOE) F = __fma_rn(__dmul_rn(-0.5, mu), vise2, F);
            }
            if (c == RHOE) F = __fma_rn(-kc, therm, F);
            if (c >= NCONS) {
                const int s = c - NCONS;
                const double Dh = face_diffusivity(P, s, vf[oL], vf[oR]);
                F = __fma_rn(-fp.mul(Dh, fp.sub(S.p[oR + sc * S.ns], S.p[oL + sc * S.ns])), B.idx[d], F);
            }
            O.p[qo + c * O.ns] = F;
            if (U.p) U.p[qu + sc * U.ns] = F;
        }
        if (U.p)
            for (int z = NCONS; z < NFLO; ++z) U.p[qu + z * U.ns] = 0.0;
        return;
    }
    // orders 4, 5 (and the species-only branch of orders 1, 2): what the flux
    // pass of this face reads
    const Fab& F = B.fs[d];
    double* q = F.p + F.off(f.i, f.j, f.k);
    q[FS_FLAGS * F.ns] = __longlong_as_double((active ? 1 : 0) | ((P.do_ns && fallback) ? 2 : 0));  // bit pattern
    q[FS_MH * F.ns] = 0.0;
    q[FS_THERM * F.ns] = fp.mul(kc, therm);
    if (active) {
        q[FS_LAMBDA * F.ns] = lam;
#pragma unroll
        for (int a = 0; a < 3; ++a) q[(FS_VIS + a) * F.ns] = fp.mul(mu, vis[a]);
        q[FS_VISE * F.ns] = fp.mul(__dmul_rn(0.5, mu), vise2);
    }
}

// Face t (linear index over growHi(bx, d, 1)) of direction d.
template <int NS, bool HIGH, bool ACTIVE = false>
__device__ __forceinline__ void face_body(const Fp& fp, const RhsBox& B, int d, int64_t t) {
    int lo[3] = {B.lo[0], B.lo[1], B.lo[2]}, len[3];
    for (int e = 0; e < 3; ++e) len[e] = B.hi[e] - B.lo[e] + 1 + (e == d);
    const int64_t nf = (int64_t)len[0] * len[1] * len[2];
    if (t >= nf) return;
    face_body_at<NS, HIGH, false, ACTIVE>(fp, B, d, delinear(t, lo, len));
}

// ---------------------------------------------------------------------------
// flux_kernel: per (face, component) along d
// ---------------------------------------------------------------------------
// WENO5 in the reference's candidate form (four divisions per edge), and the
// species convection without Navier-Stokes terms.
__device__ __forceinline__ void flux_body(const RhsBox& B, int d, int c, int64_t t) {
    int lo[3] = {B.lo[0], B.lo[1], B.lo[2]}, len[3];
    for (int e = 0; e < 3; ++e) len[e] = B.hi[e] - B.lo[e] + 1 + (e == d);
    const int64_t nf = (int64_t)len[0] * len[1] * len[2];
    if (t >= nf) return;  // c: advected component 0..4, 5.. = species
    const Idx3 f = delinear(t, lo, len);
    const DevParams& P = c_P;
    const Fab& S = B.sb;
    const int sc = (c < NCONS) ? c : c + (NFLO - NCONS);  // state component
    const int64_t sd = (d == 0) ? 1 : (d == 1) ? S.js : S.ks;
    const int64_t oR = S.off(f.i, f.j, f.k);
    const int64_t oL = oR - sd;
    const Fab& FS = B.fs[d];
    const int64_t qf = FS.off(f.i, f.j, f.k);
    const int flags = (int)__double_as_longlong(FS.p[qf + FS_FLAGS * FS.ns]);
    const bool active = flags & 1, fallback = flags & 2;
    const double* u = S.p + sc * S.ns;

    double F = 0.0;
    if (P.do_ns) {
        if (active) {
            const Fab& X = B.aux;
            const int64_t xd = (d == 0) ? 1 : (d == 1) ? X.js : X.ks;
            const int64_t xR = X.off(f.i, f.j, f.k);
            const double lam = FS.p[qf + FS_LAMBDA * FS.ns];
            double us[6], fl[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                int qq = q - 3;
                if (fallback) qq = (q < 3) ? -1 : 0;  // first-order stencil (:233-249)
                const int64_t os = oR + qq * sd, ox = xR + qq * xd;
                us[q] = u[os];
                const double rho = S.p[os + RHO * S.ns];
                const double vd = X.p[ox + (AUX_VX + d) * X.ns];
                const double va = (c >= 1 && c <= 3) ? X.p[ox + (AUX_VX + c - 1) * X.ns] : 0.0;
                const double p = X.p[ox + AUX_PF * X.ns];
                const double E = S.p[os + RHOE * S.ns];
                fl[q] = euler_flux(c, d, us[q], rho, va, vd, p, E);
            }
            double fp, fm, up, um;
            weno_face(fl, fp, fm);
            weno_face(us, up, um);
            const double fh = 0.5 * (fp + lam * up) + 0.5 * (fm - lam * um);
            F = (c < NCONS) ? fh : P.advect_flag[c - NCONS] * fh;
            if (c >= RHOU && c <= RHOW) F -= FS.p[qf + (FS_VIS + c - 1) * FS.ns];
            if (c == RHOE) F -= FS.p[qf + FS_VISE * FS.ns];
        }
        if (c == RHOE) F -= FS.p[qf + FS_THERM * FS.ns];
    } else if (c >= NCONS) {
        // species convection without Navier-Stokes (compute_flux_3d.H:382-421);
        // the limited states reduce to first order (by-value limiter, :69-83)
        const double* vfp = S.p + VFRAC * S.ns;
        const double* Vd = S.p + (VELX + d) * S.ns;
        double velface = 0.5 * (Vd[oL] + Vd[oR]);
        if (P.species_in_solid) {
            const double w = (vfp[oL] < 1.0) ? 0.0 : 1.0;  // both weights test the left cell (:410-411)
            velface = (w * Vd[oL] + w * Vd[oR]) / ((w + w) + kTiny);
        }
        F = P.advect_flag[c - NCONS] *
            ((0.5 * (velface + fabs(velface))) * u[oL] + (0.5 * (velface - fabs(velface))) * u[oR]);
    }
    if (c >= NCONS) {
        // species diffusion (compute_flux_3d.H:425-428)
        const int s = c - NCONS;
        const double* vfp = S.p + VFRAC * S.ns;
        const double Dh = face_diffusivity(P, s, vfp[oL], vfp[oR]);
        F -= (Dh * (u[oR] - u[oL])) * B.idx[d];
    }
    const Fab& O = B.flx[d];
    O.p[O.off(f.i, f.j, f.k) + c * O.ns] = F;
    if (B.uflux[d].p) {
        const Fab& U = B.uflux[d];
        const int64_t qu = U.off(f.i, f.j, f.k);
        U.p[qu + sc * U.ns] = F;
        if (c == 0)
            for (int z = NCONS; z < NFLO; ++z) U.p[qu + z * U.ns] = 0.0;
    }
}

// ---------------------------------------------------------------------------
// update_kernel: per (cell, component): divergence, masking, RK stage
// ---------------------------------------------------------------------------
// One component n of the valid cell x (volume fraction vfrac): the body of
// both launch shapes below, so they round identically.
__device__ __forceinline__ void update_one(const Fp& fp, const RhsBox& B, int stage, double dt, int n, const Idx3& x,
                                           double vfrac) {
    const DevParams& P = c_P;
    const bool advected = (n < NCONS) || (n >= NFLO);
    if (!advected && is_finite_bits(dt) && __double_as_longlong(dt) >= 0) {
        // A component without a flux (velocities, pressure, temperature,
        // density, vfrac) has the rate +0 exactly, so for a finite dt >= +0
        // dt * ds = +0 and v + dt * ds = v + 0 (plus_zero): the same bits
        // without the two FP64 operations.  n and dt are uniform over a block, so this is a branch
        // of whole warps, not a predicated path.
        if (B.dsdt.p) B.dsdt(x.i, x.j, x.k, n) = 0.0;
        if (stage == 1) {
            B.snew(x.i, x.j, x.k, n) = plus_zero(B.sb(x.i, x.j, x.k, n));
        } else if (stage == 2) {
            double v = plus_zero(B.snew(x.i, x.j, x.k, n));
            v = fp.add(v, mul(3.0, B.sold(x.i, x.j, x.k, n)));
            B.snew(x.i, x.j, x.k, n) = mul(v, 0.25);
        } else if (stage == 3) {
            double v = plus_zero(B.snew(x.i, x.j, x.k, n));
            v = fp.add(B.sold(x.i, x.j, x.k, n), mul(2.0, v));
            B.snew(x.i, x.j, x.k, n) = mul(v, kThird);
        }
        return;
    }
    double ds = 0.0;
    if (advected) {
        const int c = (n < NCONS) ? n : n - (NFLO - NCONS);
        const Fab &Fx = B.flx[0], &Fy = B.flx[1], &Fz = B.flx[2];
        const int64_t ox = Fx.off(x.i, x.j, x.k) + c * Fx.ns;
        const int64_t oy = Fy.off(x.i, x.j, x.k) + c * Fy.ns;
        const int64_t oz = Fz.off(x.i, x.j, x.k) + c * Fz.ns;
        // explicit FMAs: every compiled copy of this body rounds the same way
        ds = __fma_rn(fp.sub(Fz.p[oz], Fz.p[oz + Fz.ks]), B.idx[2],
                      __fma_rn(fp.sub(Fy.p[oy], Fy.p[oy + Fy.js]), B.idx[1],
                               mul(fp.sub(Fx.p[ox], Fx.p[ox + 1]), B.idx[0])));
        ds = plus_zero(ds);  // + source (compute_fluid_source is zero)
    }
    const int nnull = (P.species_in_solid == 1) ? NFLO : NFLO + P.nspec;
    // vfrac tests and the NaN test on the integer pipe
    if (n != RHOE) {
        if (n < nnull && below_one(vfrac)) ds = 0.0;
    } else if (!P.conj_ht) {
        if (below_one(vfrac)) ds = 0.0;
    } else if (is_positive(vfrac) && below_one(vfrac)) {
        ds = 0.0;
    }
    if (is_nan(ds)) raise_status(MFG_STATUS_NAN);
    if (B.dsdt.p) B.dsdt(x.i, x.j, x.k, n) = ds;
    // The stage algebra of the advected components with fused multiply-adds
    // (one rounding less per product than the reference's separate ones, 3
    // instead of 5 FP64 operations in stages 2 and 3); the components without
    // a flux above keep the reference's rounding, so the volume fraction and
    // the cut-cell classification it drives evolve exactly as there.
    if (stage == 1) {
        B.snew(x.i, x.j, x.k, n) = __fma_rn(dt, ds, B.sb(x.i, x.j, x.k, n));
    } else if (stage == 2) {
        double v = __fma_rn(dt, ds, B.snew(x.i, x.j, x.k, n));
        v = __fma_rn(3.0, B.sold(x.i, x.j, x.k, n), v);
        B.snew(x.i, x.j, x.k, n) = mul(v, 0.25);
    } else if (stage == 3) {
        double v = __fma_rn(dt, ds, B.snew(x.i, x.j, x.k, n));
        v = __fma_rn(2.0, v, B.sold(x.i, x.j, x.k, n));
        B.snew(x.i, x.j, x.k, n) = mul(v, kThird);
    }
}

__device__ __forceinline__ void update_body(const Fp& fp, const RhsBox& B, int stage, double dt, int n, int64_t t) {
    int lo[3] = {B.lo[0], B.lo[1], B.lo[2]}, len[3];
    for (int e = 0; e < 3; ++e) len[e] = B.hi[e] - B.lo[e] + 1;
    const int64_t nc = (int64_t)len[0] * len[1] * len[2];
    if (t >= nc) return;  // n: state component
    const Idx3 x = delinear(t, lo, len);
    const bool advected = (n < NCONS) || (n >= NFLO);
    // the flux-less components' fast path reads no volume fraction
    update_one(fp, B, stage, dt, n, x, advected ? B.sb(x.i, x.j, x.k, VFRAC) : 0.0);
}


// ---------------------------------------------------------------------------
// WENO5 column sweep (order 5 with Navier-Stokes terms, one-division mode):
// one thread walks a segment of faces along d for one component, keeping the
// per-cell parts of the reconstruction in registers.  FP64 issue bounds it
// (GB300 issues 2 FP64 operations per SM and cycle), so the form below is the
// one with the fewest FP64 operations, about 19 per (face, component).
//
// The WENO5-JS edges (flux_schemes.H:373-446) in second differences.  With
// cell differences D and t_m = v_{m-1} - 2 v_m + v_{m+1}, the linear weights
// 1 : 6 : 3 and the nonlinear weights w2 + w1 + w0 = 1, both edges of face f
// are the mean of its two cells less a sixth of a correction,
//   left  P = w2 (3 t_{f-1} - 2 t_{f-2}) + w1 t_{f-1} + w0 t_f
//           = t_{f-1} + 2 w2 (t_{f-1} - t_{f-2}) + w0 (t_f - t_{f-1}),
//   right = the same mirrored,
// (each candidate polynomial written about the mean, with w2 + w1 + w0 = 1),
// so the local Lax-Friedrichs flux needs the fluxes' mean and the corrections
// only: the state's mean cancels.  Rounding errors of the reconstruction then
// scale with the differences instead of the values: two to five times smaller
// against 80-bit arithmetic than the candidate form where the values are at least
// as large.  Beside a front, where the differences are 2^6 and more times the
// face's values, they would be larger than the flux in the end, and the face takes
// the candidates (weno_front, weno_front_llf): the test, on the integer pipe, and
// the faces it finds cost 2.5% of the 128^3 Taylor-Green step and 4% of a 64^3
// right-hand side.
//   The right edge of face m and the left edge of face m + 1 lie in cell m and
// see the same five cells, so they share the products of their weights.
//   The weights are ratios of positive numbers: mfg_weno_weights.cuh forms
// them in 64-bit fixed point on the integer pipe (560 cycles per warp, cell
// and quantity, in the shadow of about 800 on the FP64 pipe).
// Fluxes of a 64^3 box with 10 components, per right-hand side: 2.34 ms in the
// candidate form (130 FP64 operations per face and component, one division per
// edge), 1.29 ms in second differences with FP64 weights (75 operations), 0.57 ms
// with the fixed-point weights (23), 0.42 ms with the near weights added in fixed
// point and fewer integer products (19), 0.44 ms with the faces beside fronts.
// ---------------------------------------------------------------------------
constexpr int SWEEP_SEG = 32;  // longest face segment per thread (batched launches)

__device__ __forceinline__ double weight_of(uint64_t bits) { return __longlong_as_double((long long)bits); }
__device__ __forceinline__ WenoInd weno_ind(double Dm, double Dp) {
    return weno_ind(weno_diff((uint64_t)__double_as_longlong(Dm)), weno_diff((uint64_t)__double_as_longlong(Dp)));
}

// Transverse directions of a sweep along d (the first one is x when d != 0,
// so consecutive threads read consecutive addresses).
__host__ __device__ __forceinline__ void sweep_dirs(int d, int& a, int& b) {
    a = (d == 0) ? 1 : 0;
    b = (d == 2) ? 1 : 2;
}

__host__ __device__ __forceinline__ int sweep_nseg(const RhsBox& B, int d, int seg) {
    const int nf = B.hi[d] - B.lo[d] + 2;
    return (nf + seg - 1) / seg;
}

__host__ __device__ __forceinline__ int64_t sweep_items(const RhsBox& B, int d, int seg = SWEEP_SEG) {
    int a, b;
    sweep_dirs(d, a, b);
    return (int64_t)(B.hi[a] - B.lo[a] + 1) * (B.hi[b] - B.lo[b] + 1) * sweep_nseg(B, d, seg);
}

// What the WENO5 flux of component c along d reads and writes, as plain
// pointers and strides held in registers (the batched launches take the box
// from device memory, which the stores would have the compiler read again).
struct Flux5Ctx {
    const double *u, *m, *v, *p, *vf;  // state component; momentum, velocity along d; pressure; volume fraction
    const double* fs;                  // face scalars (component stride fns)
    int64_t fns;
    double* out;    // flux
    double* reg;    // flux array of the caller (component 0), or null
    int64_t rns, rsc;
    int kind;       // 0 density, 1 energy, 2 momentum along d, 3 other
    int c;
    double half;    // scale of the flux sum: 1/2 (order 4: 1/12), times the advection flag of a species
    double idx, kd; // 1/dx along d, and that times the diffusivity where it is constant
};

__device__ __forceinline__ Flux5Ctx flux5_ctx(const RhsBox& B, int d, int c) {
    Flux5Ctx x;
    const Fab &S = B.sb, &X = B.aux, &F = B.fs[d], &O = B.flx[d], &U = B.uflux[d];
    const int sc = (c < NCONS) ? c : c + (NFLO - NCONS);
    x.u = S.p + sc * S.ns;
    x.m = S.p + (RHOU + d) * S.ns;
    x.vf = S.p + VFRAC * S.ns;
    x.v = X.p + (AUX_VX + d) * X.ns;
    x.p = X.p + AUX_PF * X.ns;
    x.fs = F.p;
    x.fns = F.ns;
    x.out = O.p + c * O.ns;
    x.reg = U.p;
    x.rns = U.ns;
    x.rsc = sc * U.ns;
    x.kind = (c == RHO) ? 0 : (c == RHOE) ? 1 : (c == 1 + d) ? 2 : 3;
    x.c = c;
    x.idx = B.idx[d];
    x.half = (c < NCONS) ? 0.5 : __dmul_rn(0.5, c_P.advect_flag[c - NCONS]);
    x.kd = (c < NCONS) ? 0.0 : __dmul_rn(c_P.diff_hm[c - NCONS], x.idx);
    return x;
}

// State and Euler flux of one cell (state offset os, scratch offset ox;
// consprim_funcs.H:48-81 with a unit normal): the density flux is the momentum
// itself, the others the conserved value times the normal velocity, plus the
// pressure.
__device__ __forceinline__ void flux5_cell(const Fp& fp, const Flux5Ctx& x, int64_t os, int64_t ox, double& u,
                                           double& f) {
    u = x.u[os];
    if (x.kind == 0)
        f = x.m[os];
    else if (x.kind == 1)
        f = fp.mul(fp.add(u, x.p[ox]), x.v[ox]);
    else if (x.kind == 2)
        f = __fma_rn(u, x.v[ox], x.p[ox]);
    else
        f = fp.mul(u, x.v[ox]);
}

// Twice the local Lax-Friedrichs flux of a regular face: fsum = f_L + f_R, C
// the sum of the two edges' corrections of the Euler flux, U the difference of
// those of the state.
__device__ __forceinline__ double weno_llf(double lam, double fsum, double C, double U) {
    return __fma_rn(-1.0 / 6.0, __fma_rn(lam, U, C), fsum);
}

// C and U of one face between the cells L and R, with t the cells' second
// differences, g = t_R - t_L, gL and gR the third differences on its two sides
// and the edges' corrections
//   P_L = t_L + farL2 gL + nearL g,   P_R = t_R - nearR g - farR2 gR:
// the two near weights share their third difference and t_L - t_R is -g, so
// they are added in fixed point, with one conversion and one multiply-add for
// both (P_L and P_R apart: two more FP64 operations for C, three for U).
// sumL = t_L + farL2 gL for C, farL2 gL for U.
template <bool STATE>
__device__ __forceinline__ double weno_pair(const Fp& fp, double sumL, int64_t qL, const WenoWeights& wR, double g,
                                            double gR, double tR) {
    const int64_t q = STATE ? (qL + wR.qR) - ((int64_t)1 << 62) : qL - wR.qR;
    const double m = weight_of(signed_weight_bits(q)), far = weight_of(wR.farR2);
    if (STATE) return __fma_rn(far, gR, __fma_rn(m, g, sumL));
    return __fma_rn(-far, gR, __fma_rn(m, g, fp.add(sumL, tR)));
}

// Twice the flux of a first-order face near the immersed boundary
// (compute_flux_3d.H:233-249), weno_collapsed.
__device__ __forceinline__ double weno_llf_collapsed(const Fp& fp, double lam, double fsum, double D) {
    const double W = weight_of(weight_bits(weno_collapsed(weno_diff((uint64_t)__double_as_longlong(D))).W, 0));
    return __fma_rn(-fp.mul(lam, D), W, fsum);
}

// Twice the local Lax-Friedrichs flux of a regular face beside a front
// (weno_front): both edges of the state and of its Euler flux as weighted
// candidates, from the six cells read again (os, ox: the face's right cell; sd,
// xd: the strides along d).
__device__ __forceinline__ double weno_front_llf(const Fp& op, const Flux5Ctx& x, int64_t os, int64_t sd, int64_t ox,
                                                 int64_t xd, double lam) {
    double us[6], fl[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) flux5_cell(op, x, os + (q - 3) * sd, ox + (q - 3) * xd, us[q], fl[q]);
    const double up = weno_front_edge(us[0], us[1], us[2], us[3], us[4]);
    const double um = weno_front_edge(us[5], us[4], us[3], us[2], us[1]);
    const double fp = weno_front_edge(fl[0], fl[1], fl[2], fl[3], fl[4]);
    const double fm = weno_front_edge(fl[5], fl[4], fl[3], fl[2], fl[1]);
    return mul(op.add(__fma_rn(lam, up, fp), __fma_rn(-lam, um, fm)), 1.0 / 6.0);  // the edges come six times
}

// Complete flux of one face (the sweep and the per-face form share it, so
// they agree bitwise), stored: fh2 times x.half is the hyperbolic flux where
// active (the half, the advection flag and the viscous term take one operation),
// D = u_R - u_L, oL/oR the face's cells, qf, qo, qr its offsets in the face scalars,
// the flux scratch and the caller's flux array.
__device__ __forceinline__ void flux5_finish(const Fp& fp, const Flux5Ctx& x, bool active, double fh2, double D,
                                             int64_t oL, int64_t oR, int64_t qf, int64_t qo, int64_t qr) {
    const DevParams& P = c_P;
    const int c = x.c;
    double F = 0.0;
    if (active) {
        if (c >= RHOU && c <= RHOE)
            F = __fma_rn(x.half, fh2, -x.fs[qf + (c == RHOE ? FS_VISE : FS_VIS + c - 1) * x.fns]);
        else
            F = fp.mul(x.half, fh2);
    }
    if (c == RHOE) F = fp.sub(F, x.fs[qf + FS_THERM * x.fns]);
    if (c >= NCONS) {  // species diffusion (compute_flux_3d.H:425-428)
        const int s = c - NCONS;
        const double k = (P.diff_mode[s] == MFG_TRANSPORT_CONST)
                             ? x.kd
                             : fp.mul(face_diffusivity(P, s, x.vf[oL], x.vf[oR]), x.idx);
        F = __fma_rn(-k, D, F);
    }
    x.out[qo] = F;
    if (x.reg) {
        x.reg[qr + x.rsc] = F;
        if (c == 0)
            for (int z = NCONS; z < NFLO; ++z) x.reg[qr + z * x.rns] = 0.0;
    }
}

// Per-face form (for launches too small to fill the GPU with column
// segments): one thread per (face, component) builds its stencil itself.
__device__ __forceinline__ void flux5_face_body(const Fp& fp, const RhsBox& B, int d, int c, int64_t t) {
    int len[3];
    for (int e = 0; e < 3; ++e) len[e] = B.hi[e] - B.lo[e] + 1 + (e == d);
    if (t >= (int64_t)len[0] * len[1] * len[2]) return;
    const Idx3 f = delinear(t, B.lo, len);
    const Flux5Ctx x = flux5_ctx(B, d, c);
    const int64_t sd = (d == 0) ? 1 : (d == 1) ? B.sb.js : B.sb.ks;
    const int64_t xd = (d == 0) ? 1 : (d == 1) ? B.aux.js : B.aux.ks;
    const int64_t oR = B.sb.off(f.i, f.j, f.k), xR = B.aux.off(f.i, f.j, f.k);
    const int64_t qf = B.fs[d].off(f.i, f.j, f.k);
    const bool advected = c < NCONS || c_P.advect_flag[c - NCONS] != 0.0;  // else diffusion only
    const int flags = advected ? (int)__double_as_longlong(x.fs[qf + FS_FLAGS * x.fns]) & 3 : 0;
    double fh = 0.0, D;
    if (flags == 1) {
        double ru[6], rf[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) flux5_cell(fp, x, oR + (q - 3) * sd, xR + (q - 3) * xd, ru[q], rf[q]);
        double cu[2];  // C of the Euler flux, U of the state
        int top[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double* r = h ? ru : rf;
            double dd[5], tt[4];
#pragma unroll
            for (int q = 0; q < 5; ++q) dd[q] = fp.sub(r[q + 1], r[q]);
#pragma unroll
            for (int q = 0; q < 4; ++q) tt[q] = fp.sub(dd[q + 1], dd[q]);
            const double g0 = fp.sub(tt[1], tt[0]), g1 = fp.sub(tt[2], tt[1]), g2 = fp.sub(tt[3], tt[2]);
            const WenoInd i0 = weno_ind(dd[0], dd[1]), i1 = weno_ind(dd[1], dd[2]), i2 = weno_ind(dd[2], dd[3]),
                          i3 = weno_ind(dd[3], dd[4]);
            const WenoWeights wl = weno_weights(i0.dB, i0.eB, i1.dC, i1.eC, i2.dA, i2.eA);
            const WenoWeights wr = weno_weights(i1.dB, i1.eB, i2.dC, i2.eC, i3.dA, i3.eA);
            cu[h] = h ? weno_pair<true>(fp, fp.mul(weight_of(wl.farL2), g0), wl.qL, wr, g1, g2, tt[2])
                      : weno_pair<false>(fp, __fma_rn(weight_of(wl.farL2), g0, tt[1]), wl.qL, wr, g1, g2, tt[2]);
            top[h] = imax(imax(i0.eB, i1.eB), imax(i2.eB, i3.eB));
            if (h) D = dd[2];
        }
        const double lam = x.fs[qf + FS_LAMBDA * x.fns];
        fh = weno_front(top[0], top[1], x.kind == 2, rf[2], rf[3], ru[2], ru[3], lam)
                 ? weno_front_llf(fp, x, oR, sd, xR, xd, lam)
                 : weno_llf(lam, fp.add(rf[2], rf[3]), cu[0], cu[1]);
    } else if (flags & 1) {
        double uL, uR, fL, fR;
        flux5_cell(fp, x, oR - sd, xR - xd, uL, fL);
        flux5_cell(fp, x, oR, xR, uR, fR);
        D = fp.sub(uR, uL);
        fh = weno_llf_collapsed(fp, x.fs[qf + FS_LAMBDA * x.fns], fp.add(fL, fR), D);
    } else {
        D = fp.sub(x.u[oR], x.u[oR - sd]);
    }
    flux5_finish(fp, x, flags & 1, fh, D, oR - sd, oR, qf, B.flx[d].off(f.i, f.j, f.k),
                 x.reg ? B.uflux[d].off(f.i, f.j, f.k) : 0);
}

// Order 4, central with dissipation (the reference's central_with_diss_flux:
// (7 (f_L + f_R) - f_LL - f_RR - lam dissfactor (3 u_R - 3 u_L - u_RR + u_R))
// / 12, its twelfth rounded to ten digits): one thread per (face, component), the
// four cells it reads as the order-5 sweep takes them (one or two FP64 operations
// each, against six cells of the general Euler flux before), half, flag and viscous
// term in one multiply-add: about 16 FP64 operations against 60 (right-hand side of
// 57x64x33 cells 287 -> 217 us).  The outer cells are added to the dissipation before
// they leave seven times the inner sum: one rounding of that size, where the terms in
// turn had two to four.
__device__ __forceinline__ void flux4_body(const Fp& fp, const RhsBox& B, int d, int c, int64_t t) {
    int len[3];
    for (int e = 0; e < 3; ++e) len[e] = B.hi[e] - B.lo[e] + 1 + (e == d);
    if (t >= (int64_t)len[0] * len[1] * len[2]) return;
    const Idx3 f = delinear(t, B.lo, len);
    Flux5Ctx x = flux5_ctx(B, d, c);
    x.half = (c < NCONS) ? kTwelveth : __dmul_rn(kTwelveth, c_P.advect_flag[c - NCONS]);
    const int64_t sd = (d == 0) ? 1 : (d == 1) ? B.sb.js : B.sb.ks;
    const int64_t xd = (d == 0) ? 1 : (d == 1) ? B.aux.js : B.aux.ks;
    const int64_t oR = B.sb.off(f.i, f.j, f.k), xR = B.aux.off(f.i, f.j, f.k);
    const int64_t qf = B.fs[d].off(f.i, f.j, f.k);
    const int flags = (int)__double_as_longlong(x.fs[qf + FS_FLAGS * x.fns]);
    double S = 0.0, D;
    if (flags & 1) {
        const double lam = __dmul_rn(x.fs[qf + FS_LAMBDA * x.fns], c_P.dissfactor);
        double u[4], fl[4];  // cells LL, L, R, RR
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int at = (flags & 2) ? (q < 2 ? -1 : 0) : q - 2;  // first-order stencil (:233-249)
            flux5_cell(fp, x, oR + at * sd, xR + at * xd, u[q], fl[q]);
        }
        D = fp.sub(u[2], u[1]);
        const double outer = __fma_rn(lam, __fma_rn(3.0, D, fp.sub(u[2], u[3])), fp.add(fl[0], fl[3]));
        S = __fma_rn(7.0, fp.add(fl[1], fl[2]), -outer);
    } else {
        D = fp.sub(x.u[oR], x.u[oR - sd]);
    }
    flux5_finish(fp, x, flags & 1, S, D, oR - sd, oR, qf, B.flx[d].off(f.i, f.j, f.k),
                 x.reg ? B.uflux[d].off(f.i, f.j, f.k) : 0);
}

// Carried from face to face for one of the two reconstructed quantities (the
// state or its Euler flux): v0, v1 = cells f, f+1; D = v1 - v0; t_f and g =
// t_f - t_{f-1}; the indicators of the centres f-1 (B) and f (B, C); the left
// cell's part of C or U at this face (weno_pair) and its near weight.
struct WenoRun {
    double v0, v1, D;
    double t0, g, sumL;
    int64_t qL;
    uint64_t dBm, dB0, dC0;
    int eBm, eB0, eC0, eBp;  // eBp: of centre f-2
};

// Adds centre f+1 (Dn = v_{f+2} - v_{f+1}): returns C or U of face f, in top the
// largest eB of its four centres (weno_front), and moves the run to face f+1.
template <bool STATE>
__device__ __forceinline__ double weno_next(const Fp& fp, WenoRun& r, double D, double Dn, int& top) {
    const WenoInd c = weno_ind(D, Dn);
    top = imax(imax(r.eBp, r.eBm), imax(r.eB0, c.eB));
    r.eBp = r.eBm;
    const WenoWeights w = weno_weights(r.dBm, r.eBm, r.dC0, r.eC0, c.dA, c.eA);
    const double t = fp.sub(Dn, D), gp = fp.sub(t, r.t0);
    const double res = weno_pair<STATE>(fp, r.sumL, r.qL, w, r.g, gp, r.t0);
    r.sumL = STATE ? fp.mul(weight_of(w.farL2), r.g) : __fma_rn(weight_of(w.farL2), r.g, r.t0);
    r.qL = w.qL;
    r.t0 = t;
    r.g = gp;
    r.dBm = r.dB0;
    r.eBm = r.eB0;
    r.dB0 = c.dB;
    r.eB0 = c.eB;
    r.dC0 = c.dC;
    r.eC0 = c.eC;
    return res;
}

// Starts the run at face f: va .. vL = cells f-3, f-2, f-1.
template <bool STATE>
__device__ __forceinline__ void weno_prime(const Fp& fp, WenoRun& r, double va, double vb, double vL) {
    const double d0 = fp.sub(vb, va), d1 = fp.sub(vL, vb), d2 = fp.sub(r.v0, vL);
    const WenoInd c0 = weno_ind(d0, d1), c1 = weno_ind(d1, d2);
    const double ta = fp.sub(d1, d0);
    r.t0 = fp.sub(d2, d1);
    r.g = fp.sub(r.t0, ta);
    r.sumL = 0.0;
    r.qL = 0;
    r.eBp = 0;
    r.dBm = c0.dB;
    r.eBm = c0.eB;
    r.dB0 = c1.dB;
    r.eB0 = c1.eB;
    r.dC0 = c1.dC;
    r.eC0 = c1.eC;
    int top;
    weno_next<STATE>(fp, r, d2, r.D, top);
}

// Column segment t of a sweep: its first face f (indices) and its number of faces.
__device__ __forceinline__ int sweep_segment(const RhsBox& B, int d, int64_t t, int seglen, Idx3& f) {
    int ta, tb;
    sweep_dirs(d, ta, tb);
    const int na = B.hi[ta] - B.lo[ta] + 1, nb = B.hi[tb] - B.lo[tb] + 1;
    const int64_t ncol = (int64_t)na * nb;
    const int seg = (int)(t / ncol);
    const int64_t col = t - (int64_t)seg * ncol;
    const int nf = B.hi[d] - B.lo[d] + 2;
    const int nseg = sweep_nseg(B, d, seglen);
    const int per = (nf + nseg - 1) / nseg;
    const int f0 = B.lo[d] + seg * per;
    const int ia = B.lo[ta] + (int)(col % na), ib = B.lo[tb] + (int)(col / na);
    f.i = (d == 0) ? f0 : ia;
    f.j = (d == 0) ? ia : (d == 1) ? f0 : ib;
    f.k = (d == 2) ? f0 : ib;
    return min(per, B.lo[d] + nf - f0);
}

// The faces of a column segment that are beside a front (bit q: the face q before
// the last), done again by the candidates.  Apart from the walk and not inlined:
// it shares no registers with it (inside the loop the kernel spilled 200 bytes,
// after it 50, the batched one 500 against 270), and few segments come here.
__device__ __noinline__ void flux5_fronts(const RhsBox& B, int d, int c, int64_t t, int seglen, unsigned fronts) {
    const Fp fp(0);  // few lanes of a warp are here: no shuffle
    Idx3 f;
    int n = sweep_segment(B, d, t, seglen, f);
    const Flux5Ctx x = flux5_ctx(B, d, c);
    const int64_t sd = (d == 0) ? 1 : (d == 1) ? B.sb.js : B.sb.ks;
    const int64_t xd = (d == 0) ? 1 : (d == 1) ? B.aux.js : B.aux.ks;
    const int64_t fd = (d == 0) ? 1 : (d == 1) ? B.fs[d].js : B.fs[d].ks;
    const int64_t rd = (d == 0) ? 1 : (d == 1) ? B.uflux[d].js : B.uflux[d].ks;
    const int64_t o0 = B.sb.off(f.i, f.j, f.k), a0 = B.aux.off(f.i, f.j, f.k), q0 = B.fs[d].off(f.i, f.j, f.k);
    const int64_t r0 = x.reg ? B.uflux[d].off(f.i, f.j, f.k) : 0;
    for (; fronts; fronts &= fronts - 1) {
        const int m = n - __ffs(fronts);
        const int64_t o = o0 + m * sd, q = q0 + m * fd;
        const double fh = weno_front_llf(fp, x, o, sd, a0 + m * xd, xd, x.fs[q + FS_LAMBDA * x.fns]);
        flux5_finish(fp, x, true, fh, fp.sub(x.u[o], x.u[o - sd]), o - sd, o, q, q, r0 + m * rd);
    }
}

__device__ __forceinline__ void flux5_sweep_body(const Fp& fp, const RhsBox& B, int d, int c, int64_t t,
                                                 int seglen = SWEEP_SEG) {
    if (t >= sweep_items(B, d, seglen)) return;
    Idx3 f0;
    int left = sweep_segment(B, d, t, seglen, f0);  // faces to do
    if (left <= 0) return;
    const int i = f0.i, j = f0.j, k = f0.k;
    const Flux5Ctx x = flux5_ctx(B, d, c);
    const int64_t sd = (d == 0) ? 1 : (d == 1) ? B.sb.js : B.sb.ks;
    const int64_t xd = (d == 0) ? 1 : (d == 1) ? B.aux.js : B.aux.ks;
    // the face scalars and the flux scratch have the same extents
    const int64_t fd = (d == 0) ? 1 : (d == 1) ? B.fs[d].js : B.fs[d].ks;
    const int64_t rd = (d == 0) ? 1 : (d == 1) ? B.uflux[d].js : B.uflux[d].ks;
    int64_t oR = B.sb.off(i, j, k);  // right cell of the current face
    int64_t xR = B.aux.off(i, j, k);
    int64_t qf = B.fs[d].off(i, j, k);
    int64_t qr = x.reg ? B.uflux[d].off(i, j, k) : 0;
    if (c >= NCONS && c_P.advect_flag[c - NCONS] == 0.0) {  // not advected: diffusion only
        for (; left > 0; --left, oR += sd, qf += fd, qr += rd)
            flux5_finish(fp, x, false, 0.0, fp.sub(x.u[oR], x.u[oR - sd]), oR - sd, oR, qf, qf, qr);
        return;
    }
    // Cells f-1 .. f+1 to start with; the WENO parts are built only where a
    // face of the warp needs them: faces on the solid side of the immersed
    // boundary (no hyperbolic flux) and first-order fallback faces use the cell
    // values alone.  A lane at such a face beside a regular one advances its run
    // with the others, in slots that divergence would leave idle, rather than
    // start it again (three centres) at its own next regular face (the run is a
    // function of the cells alone, so the numbers do not depend on it): fluxes of
    // the 64^3 catalyst step 4.45 -> 4.09 ms.
    WenoRun u, f;
    double uL, fL;
    flux5_cell(fp, x, oR - sd, xR - xd, uL, fL);
    flux5_cell(fp, x, oR, xR, u.v0, f.v0);
    flux5_cell(fp, x, oR + sd, xR + xd, u.v1, f.v1);
    double Du = fp.sub(u.v0, uL);  // u_f - u_{f-1}
    u.D = fp.sub(u.v1, u.v0);
    f.D = fp.sub(f.v1, f.v0);
    bool primed = false;
    unsigned fronts = 0;  // faces beside a front, done again below (a segment has up to 32)
    for (;;) {
        double un, fn;  // cell f+2, loaded before this face's arithmetic
        flux5_cell(fp, x, oR + 2 * sd, xR + 2 * xd, un, fn);
        const int flags = (int)__double_as_longlong(x.fs[qf + FS_FLAGS * x.fns]) & 3;
        const double Dun = fp.sub(un, u.v1), Dfn = fp.sub(fn, f.v1);
        double fh = 0.0;
        if (__any_sync(__activemask(), flags == 1)) {
            if (!primed) {
                double ua, fa, ub, fb;
                flux5_cell(fp, x, oR - 3 * sd, xR - 3 * xd, ua, fa);
                flux5_cell(fp, x, oR - 2 * sd, xR - 2 * xd, ub, fb);
                weno_prime<true>(fp, u, ua, ub, uL);
                weno_prime<false>(fp, f, fa, fb, fL);
                primed = true;
            }
            int topf, topu;
            const double C = weno_next<false>(fp, f, f.D, Dfn, topf), U = weno_next<true>(fp, u, u.D, Dun, topu);
            if (flags == 1) {
                const double lam = x.fs[qf + FS_LAMBDA * x.fns];
                fh = weno_llf(lam, fp.add(fL, f.v0), C, U);
                if (weno_front(topf, topu, x.kind == 2, fL, f.v0, uL, u.v0, lam)) fronts |= 1u;
            }
        } else {
            primed = false;
        }
        if (flags == 3) fh = weno_llf_collapsed(fp, x.fs[qf + FS_LAMBDA * x.fns], fp.add(fL, f.v0), Du);
        flux5_finish(fp, x, flags & 1, fh, Du, oR - sd, oR, qf, qf, qr);
        if (--left == 0) break;
        fronts <<= 1;
        // advance one face
        oR += sd;
        xR += xd;
        qf += fd;
        qr += rd;
        uL = u.v0;
        fL = f.v0;
        Du = u.D;
        u.v0 = u.v1;
        f.v0 = f.v1;
        u.v1 = un;
        f.v1 = fn;
        u.D = Dun;
        f.D = Dfn;
    }
    if (fronts) flux5_fronts(B, d, c, t, seglen, fronts);
}

// Work items of each phase for one box.
__host__ __device__ __forceinline__ int64_t prim_items(const RhsBox& B) {
    return (int64_t)(B.hi[0] - B.lo[0] + 7) * (B.hi[1] - B.lo[1] + 7) * (B.hi[2] - B.lo[2] + 7);
}
__host__ __device__ __forceinline__ int64_t face_items(const RhsBox& B, int d) {
    return (int64_t)(B.hi[0] - B.lo[0] + 1 + (d == 0)) * (B.hi[1] - B.lo[1] + 1 + (d == 1)) *
           (B.hi[2] - B.lo[2] + 1 + (d == 2));
}
__host__ __device__ __forceinline__ int64_t cell_items(const RhsBox& B) {
    return (int64_t)(B.hi[0] - B.lo[0] + 1) * (B.hi[1] - B.lo[1] + 1) * (B.hi[2] - B.lo[2] + 1);
}

}  // namespace
}  // namespace mfg
