// Device thermodynamics and transport for the three thermo families of the
// reference's case plugins, evaluated from the parameter tables in constant
// memory.  Operand order follows the plugins (sums over gas species in
// ascending order, divisions where the plugins divide) so the FP64 results
// track the reference's rounding.
#pragma once
#include "mfg_common.cuh"

namespace mfg {

extern __constant__ DevParams c_P;

// Temperature from (rho, p, species).  Molar: ShockTube_N2/thermo.H:58-67,
// catalystCylinder/thermo.H:54-63; mass-single: porousParticle/thermo.H:54-59;
// background gas: rxnscheme example thermo.H:61-76.
template <int NS>
__device__ __forceinline__ double thermo_t(double rho, double pres, const double* spec) {
    const DevParams& P = c_P;
    if (P.thermo_kind == MFG_THERMO_MASS_SINGLE) return pres / P.gas_R / rho;
    double sum_ci = 0.0;
    if (P.thermo_kind == MFG_THERMO_BG_GAS) {
        double sum_ciMi = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (s < P.ngas) {
                sum_ci += spec[s];
                sum_ciMi += spec[s] * P.molwt[s];
            }
        double c_bg = (rho - sum_ciMi) / P.bg_molwt;
        sum_ci += c_bg;
        return pres / (sum_ci * kRU);
    }
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < P.ngas) sum_ci += spec[s];
    return pres / (sum_ci * P.R_univ);
}

// Mixture density from the species concentrations (thermo.H get_r_from_c):
// molar, catalystCylinder/thermo.H:37-45 (gas species); mass-single,
// TaylorGreen/thermo.H:37-45 (every species); background gas, rxnscheme
// example thermo.H:20-31 (gas species + bgasconc W_bg).
template <int NS>
__device__ __forceinline__ double thermo_r_from_c(const double* spec, double bgasconc) {
    const DevParams& P = c_P;
    const int n = (P.thermo_kind == MFG_THERMO_MASS_SINGLE) ? P.nspec : P.ngas;
    double rho = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < n) rho = add(rho, mul(spec[s], P.molwt[s]));
    if (P.thermo_kind == MFG_THERMO_BG_GAS) rho = add(rho, mul(bgasconc, P.bg_molwt));
    return rho;
}

// Untracked background-gas concentration (thermo.H get_bgasconc_from_rc):
// molar 0 (catalystCylinder/thermo.H:47-52), mass-single the first species
// (TaylorGreen/thermo.H:46-53), background gas (rho - sum c W) / W_bg
// (rxnscheme example thermo.H:32-42).
template <int NS>
__device__ __forceinline__ double thermo_bgasconc(double rho, const double* spec) {
    const DevParams& P = c_P;
    if (P.thermo_kind == MFG_THERMO_MASS_SINGLE) return spec[0];
    if (P.thermo_kind != MFG_THERMO_BG_GAS) return 0.0;
    double sum_ciMi = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < P.ngas) sum_ciMi = add(sum_ciMi, mul(spec[s], P.molwt[s]));
    return __ddiv_rn(__dsub_rn(rho, sum_ciMi), P.bg_molwt);
}

// Concentration of the untracked background gas.
template <int NS>
__device__ __forceinline__ double background_conc(double rho, const double* spec) {
    const DevParams& P = c_P;
    double sum_ciMi = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < P.ngas) sum_ciMi = __fma_rn(spec[s], P.molwt[s], sum_ciMi);
    return (rho - sum_ciMi) / P.bg_molwt;
}

// Numerator and denominator of kappa = p / (rho e) = gamma - 1 of the molar and
// background-gas families: the mixture gamma less one is 1 / sum(x_k / (gamma_k -
// 1)) with mole fractions x_k (thermo.H get_gama_from_rc), and with cv_k = R /
// (gamma_k - 1) it is also p / (rho e) of T = rho e / sum(cv c), p = R T sum(c)
// (thermo.H get_p_from_rec).  The denominator is the numerator sum(c) times the
// smallest 1 / (gamma_k - 1) plus the (positive) rest: the rounding of sum(c)
// drops out of the ratio.  Against extended precision the pressure's rms error is
// 0.95 x 2^-53, on five and on eight species; the plugins' order of operations has
// 1.05 and 1.27, sums of c and of cv c on their own 1.18 and 1.30.
template <int NS>
__device__ __forceinline__ void thermo_ratio(double rho, const double* spec, double& num, double& den) {
    const DevParams& P = c_P;
    double sc = spec[0], rest = __dmul_rn(P.igd[0], spec[0]);
#pragma unroll
    for (int s = 1; s < NS; ++s)
        if (s < P.ngas) {
            sc = __dadd_rn(sc, spec[s]);
            rest = __fma_rn(P.igd[s], spec[s], rest);
        }
    if (P.thermo_kind == MFG_THERMO_BG_GAS) {
        const double c_bg = background_conc<NS>(rho, spec);
        sc = __dadd_rn(sc, c_bg);
        rest = __fma_rn(P.igd[P.ngas], c_bg, rest);
    }
    num = sc;
    den = __fma_rn(P.ig_min, sc, rest);
}

// kappa = p / (rho e) = gamma - 1: one division serves pressure, gamma and
// sound speed (14 FP64 operations for five species, against about 80 for
// the pressure twice and gamma each with its own divisions and sums).
template <int NS>
__device__ __forceinline__ double thermo_kappa(double rho, const double* spec) {
    if (c_P.thermo_kind == MFG_THERMO_MASS_SINGLE) return c_P.gm1_single;
    double n, d;
    thermo_ratio<NS>(rho, spec, n, d);
    return quot(n, d);
}

// Pressure from (rho e, rho, species).
template <int NS>
__device__ __forceinline__ double thermo_p(double rhoe, double rho, const double* spec) {
    return rhoe * thermo_kappa<NS>(rho, spec);
}

// Pressure and temperature from (rho e, rho, species): p = kappa rho e, T = rho e /
// sum(cv c), in two chains (even and odd species: fewer roundings); mass-single p =
// (gamma - 1) rho e, T = (p / rho) / R with irho = 1/rho and the reciprocal of R
// from mfg_init.
template <int NS>
__device__ __forceinline__ void thermo_pt(double rhoe, double rho, double irho, const double* spec, double& p,
                                          double& T) {
    const DevParams& P = c_P;
    p = rhoe * thermo_kappa<NS>(rho, spec);
    if (P.thermo_kind == MFG_THERMO_MASS_SINGLE) {
        T = (p * irho) * P.inv_gas_R;
        return;
    }
    double c2[2] = {0.0, 0.0};
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < P.ngas) c2[s & 1] = __fma_rn(P.cv[s], spec[s], c2[s & 1]);
    double cvs = c2[0] + c2[1];
    if (P.thermo_kind == MFG_THERMO_BG_GAS) cvs = __fma_rn(P.cv[P.ngas], background_conc<NS>(rho, spec), cvs);
    T = quot(rhoe, cvs);
}

// Mixture gamma (depends on composition only).
template <int NS>
__device__ __forceinline__ double thermo_gamma(double rho, const double* spec) {
    if (c_P.thermo_kind == MFG_THERMO_MASS_SINGLE) return c_P.gamma_single;
    return 1.0 + thermo_kappa<NS>(rho, spec);
}

// Specific internal energy from (rho, p, species).
template <int NS>
__device__ __forceinline__ double thermo_e(double rho, double pres, const double* spec) {
    const DevParams& P = c_P;
    if (P.thermo_kind == MFG_THERMO_MASS_SINGLE) return pres / (P.gamma_single - 1.0) / rho;
    if (P.thermo_kind == MFG_THERMO_BG_GAS) {
        double sum_ciMi = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (s < P.ngas) sum_ciMi += spec[s] * P.molwt[s];
        double c_bg = (rho - sum_ciMi) / P.bg_molwt;
        double temp = thermo_t<NS>(rho, pres, spec);
        double scv = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (s < P.ngas) scv += P.cv[s] * spec[s];
        scv += P.cv[P.ngas] * c_bg;
        return scv * temp / rho;
    }
    if (P.energy_form == MFG_EFORM_MASS_CV) {
        double sum_ci = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (s < P.ngas) sum_ci += spec[s];
        double temp = thermo_t<NS>(rho, pres, spec);
        double cvbar = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (s < P.ngas) cvbar += P.cvmass[s] * (spec[s] / sum_ci);
        return cvbar * temp;
    }
    double temp = thermo_t<NS>(rho, pres, spec);
    double scv = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < P.ngas) scv += P.cv[s] * spec[s];
    return scv * temp / rho;
}

// Transport coefficient: constant, or gas*vfrac + solid*(1-vfrac).
__device__ __forceinline__ double blend(int mode, double g, double s, double vf) {
    return (mode == MFG_TRANSPORT_VFRAC_BLEND) ? (g * vf + s * (1.0 - vf)) : g;
}

// 2 d1 d2 / (d1 + d2 + 1e-30)  (compute_flux_3d.H:18-22)
__device__ __forceinline__ double harmonic_mean(double d1, double d2) {
    return 2.0 * d1 * d2 / (d1 + d2 + 1e-30);
}

// Diffusivity of species s at the face between cells of volume fractions vL and
// vR: the harmonic mean of the two cells' coefficients (compute_flux_3d.H:
// 425-428).  Between two gas or two solid cells it is a constant from mfg_init
// (the blend gas vf + solid (1 - vf) is the gas or the solid value exactly); the
// blend and its division, 18 FP64 slots per species and face, remain for faces
// of cut cells.
__device__ __forceinline__ double face_diffusivity(const DevParams& P, int s, double vL, double vR) {
    if (P.diff_mode[s] == MFG_TRANSPORT_CONST || (is_one(vL) && is_one(vR))) return P.diff_hm[s];
    if (is_zero_bits(vL) && is_zero_bits(vR)) return P.diff_hms[s];
    const double g = P.diff_gas[s], so = P.diff_solid[s];
    const double dl = __fma_rn(g, vL, mul(so, sub(1.0, vL))), dr = __fma_rn(g, vR, mul(so, sub(1.0, vR)));
    return quot_mid(mul(mul(2.0, dl), dr), add(add(dl, dr), 1e-30));  // the divisor is at least 1e-30
}

}  // namespace mfg
