// Physical-boundary device code of the ghost fill (wall parity, ext_dir ghost
// state), shared by the single-level fill (mfg_fill.cu) and the multi-level
// batched fill (mfg_batch.cu).
#pragma once
#include "mfg_internal.h"
#include "mfg_physics.cuh"

namespace mfg {
namespace {

__device__ __forceinline__ bool odd_at_wall(int n) {  // Source/mflo.cpp:98-110
    return (n >= RHOU && n <= RHOW) || (n >= VELX && n <= VELZ);
}

// ext_dir ghost state (the case's externalbc functor as a parameterised template)
template <int NS>
__device__ void external_state(const mfg_extbc& E, int idir, const double* s_int, double* s_ext, int nc) {
    const int ns = c_P.nspec;
#pragma unroll
    for (int n = 0; n < NFLO + NS; ++n) s_ext[n] = 0.0;
    if (E.kind == MFG_EXT_FIXED_STATE) {
#pragma unroll
        for (int n = 0; n < NFLO + NS; ++n)
            if (n < nc) s_ext[n] = E.state[n];
        if (E.keep_interior_pres) s_ext[PRES] = s_int[PRES];
        return;
    }
    if (E.kind == MFG_EXT_SPECIES_DIRICHLET) {
#pragma unroll
        for (int n = 0; n < NFLO; ++n) s_ext[n] = s_int[n];
        if (!E.vfrac_interior) s_ext[VFRAC] = 1.0;
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (s < ns)
                s_ext[NFLO + s] = ((E.spec_zero_grad_mask >> s) & 1)
                                      ? s_int[NFLO + s]
                                      : __dsub_rn(__dmul_rn(2.0, E.spec[s]), s_int[NFLO + s]);
        return;
    }
    double spec[NS];
    double dens, pres, vel[3];
    if (E.kind == MFG_EXT_PRESSURE_INLET) {
        dens = E.dens;
        pres = E.pres;
        const double vm = sqrt((s_int[VELX] * s_int[VELX] + s_int[VELY] * s_int[VELY]) + s_int[VELZ] * s_int[VELZ]);
        vel[0] = (idir == 0) ? vm : 0.0;
        vel[1] = (idir == 1) ? vm : 0.0;
        vel[2] = (idir == 2) ? vm : 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) spec[s] = (s < ns) ? E.spec[s] : 0.0;
    } else if (E.kind == MFG_EXT_PRESSURE_OUTLET) {
        dens = s_int[DENS];
        pres = E.pres;
        vel[0] = s_int[VELX];
        vel[1] = s_int[VELY];
        vel[2] = s_int[VELZ];
#pragma unroll
        for (int s = 0; s < NS; ++s) spec[s] = (s < ns) ? s_int[NFLO + s] : 0.0;
    } else {
        dens = E.dens;
        pres = E.pres;
        vel[0] = E.vel[0];
        vel[1] = E.vel[1];
        vel[2] = E.vel[2];
#pragma unroll
        for (int s = 0; s < NS; ++s) spec[s] = (s < ns) ? E.spec[s] : 0.0;
    }
    s_ext[DENS] = dens;
    s_ext[PRES] = pres;
    s_ext[VELX] = vel[0];
    s_ext[VELY] = vel[1];
    s_ext[VELZ] = vel[2];
    s_ext[TEMP] = thermo_t<NS>(dens, pres, spec);
    s_ext[RHO] = dens;
    s_ext[RHOU] = mul(dens, vel[0]);
    s_ext[RHOV] = mul(dens, vel[1]);
    s_ext[RHOW] = mul(dens, vel[2]);
    const double ke = add(add(mul(vel[0], vel[0]), mul(vel[1], vel[1])), mul(vel[2], vel[2]));
    s_ext[RHOE] = add(mul(dens, thermo_e<NS>(dens, pres, spec)), mul(mul(0.5, dens), ke));
#pragma unroll
    for (int s = 0; s < NS; ++s)
        if (s < ns) s_ext[NFLO + s] = spec[s];
    s_ext[VFRAC] = s_int[VFRAC];
}

// Physical boundary of cell (i, j, k) of S, outside the domain in one to three
// directions.  The reference fills faces, then edges, then corners, each from
// the cell one direction further in (through an ext_dir direction first, the
// highest, otherwise the highest): here the chain is followed to the cell inside
// the domain it ends at and its steps are applied to that cell's state, the
// innermost first, so every cell is filled in one launch from cells that the
// launch does not write.  Walls change the sign of the momenta and velocities
// each, and stand before any ext_dir state in the chain.  Latency bounds it:
// three launches with one component's load and store after the other took 61 us
// per stage of a 64^3 catalyst step, this one 23 us.
template <int NS>
__device__ __forceinline__ void bc_fill(const Fab& S, const int dlo[3], const int dhi[3], const int per[3], int i,
                                        int j, int k, int nc) {
    const DevParams& P = c_P;
    const int64_t qd = S.off(i, j, k);
    int iv[3] = {i, j, k}, ext[3], next = 0;
    bool out[3], odd = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) out[d] = !per[d] && (iv[d] < dlo[d] || iv[d] > dhi[d]);
    if (!(out[0] || out[1] || out[2])) return;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        int dext = -1, dlast = -1;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (!out[d]) continue;
            dlast = d;
            if (((iv[d] < dlo[d]) ? P.bc_lo[d] : P.bc_hi[d]) == MFG_BC_EXT_DIR) dext = d;
        }
        const int ds = (dext >= 0) ? dext : dlast;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (d != ds) continue;
            const bool lo = iv[d] < dlo[d];
            const int kind = lo ? P.bc_lo[d] : P.bc_hi[d];
            if (kind == MFG_BC_EXT_DIR || kind == MFG_BC_FOEXTRAP) {
                iv[d] = lo ? dlo[d] : dhi[d];
            } else {  // wall: reflect_even, reflect_odd for momenta and velocities
                iv[d] = lo ? (2 * dlo[d] - iv[d] - 1) : (2 * dhi[d] - iv[d] + 1);
                odd = !odd;
            }
            if (kind == MFG_BC_EXT_DIR) ext[next++] = 2 * d + (lo ? 0 : 1);
            out[d] = false;
        }
    }
    const double* src = S.p + S.off(iv[0], iv[1], iv[2]);
    double* dst = S.p + qd;
    if (next == 0) {
        for (int c = 0; c < nc; c += 4) {  // four loads in flight
            double x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = (c + u < nc) ? src[(c + u) * S.ns] : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c + u < nc) dst[(c + u) * S.ns] = (odd && odd_at_wall(c + u)) ? -x[u] : x[u];
        }
        return;
    }
    double s[NFLO + NS], t[NFLO + NS];
#pragma unroll
    for (int c = 0; c < NFLO + NS; ++c) {
        s[c] = (c < nc) ? src[c * S.ns] : 0.0;
        if (odd && odd_at_wall(c)) s[c] = -s[c];
    }
    for (int q = next - 1; q >= 0; --q) {
        const int d = ext[q] >> 1;
        external_state<NS>((ext[q] & 1) ? P.ext_hi[d] : P.ext_lo[d], d, s, t, nc);
#pragma unroll
        for (int c = 0; c < NFLO + NS; ++c) s[c] = t[c];
    }
#pragma unroll
    for (int c = 0; c < NFLO + NS; ++c)
        if (c < nc) dst[c * S.ns] = s[c];
}

}  // namespace
}  // namespace mfg
