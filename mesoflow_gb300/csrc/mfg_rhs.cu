// Flow right-hand side and fused RK3 stage update for one AMReX box.
//
// Structure (per RK stage; each kernel one launch for a group of boxes,
// mfg_rhs_launch.cuh):
//   prim_kernel   per cell of grow(bx,3): velocities, pressure, eigen-pressure
//                 energy, own sound speed and gamma - 1, computed once per cell
//                 instead of once per face use (the reference re-derives them
//                 inside every face's geteulerflux / get_max_eigenvalue).
//   face_kernel   per face of growHi(bx,d,1): scheme scalars (LLF eigenvalue,
//                 AUSM+-up Mach/pressure terms), IB flags, viscous stress and
//                 heat-conduction terms.  Orders 1/2 with Navier-Stokes terms
//                 split it: face_split_kernel writes the faces on the solid
//                 side (conduction and diffusion only) and lists the others,
//                 face_list_kernel runs the flux branch over those lists, each
//                 for the three directions in one launch, so no lane of a warp
//                 idles on a solid-side face.
//   flux5_sweep_kernel  WENO5 with Navier-Stokes terms: per (column segment
//                 along d, component), the per-cell parts of the reconstruction
//                 computed once per cell and kept in registers while the thread
//                 walks the faces; species diffusion and viscous terms included,
//                 written once per face and read by both neighbouring cells.
//                 flux5_face_kernel is the per-face form for small launches.
//   flux4_kernel  per (face, component): the central scheme with dissipation.
//   flux_kernel   per (face, component): WENO5 in the reference's operation
//                 order (mfg_set_weno_mode 0), and the species convection
//                 without Navier-Stokes terms.
//   update_kernel per (cell, component): flux divergence, IB masking, NaN
//                 status, and the RK3 stage algebra.
// Semantics: compute_flux (Source/Src_3d/compute_flux_3d.H:88-430),
// update_residual (Source/Src_3d/div_3d.H:13-76), stage algebra
// (Source/mflo_evolve.cpp:276-311).
#include "mfg_rhs_launch.cuh"

namespace mfg {

__constant__ DevParams c_P;
__device__ unsigned int g_status = 0;

namespace {

bool g_face_split = true;  // mfg_set_face_compaction

}  // namespace

cudaError_t upload_params(const DevParams& h) { return cudaMemcpyToSymbol(c_P, &h, sizeof(DevParams)); }

cudaError_t read_status(unsigned* v, bool clear) {
    cudaError_t e = cudaMemcpyFromSymbol(v, g_status, sizeof(unsigned));
    if (e == cudaSuccess && clear) {
        unsigned z = 0;
        e = cudaMemcpyToSymbol(g_status, &z, sizeof(unsigned));
    }
    return e;
}

cudaError_t launch_rhs_box(const RhsBox& B, int stage, double dt, bool fast, cudaStream_t st) {
    return launch_group<1>(&B, 1, stage, dt, fast, g_face_split, st);
}

cudaError_t launch_rhs_boxes(const RhsBox* boxes, int n, int stage, double dt, bool fast, cudaStream_t st) {
    if (n == 1) return launch_rhs_box(boxes[0], stage, dt, fast, st);
    return launch_rhs_group(boxes, n, stage, dt, fast, g_face_split, st);
}

int rhs_group_count(const mfg_box* boxes, int nbox) {
    int64_t cells = 0;
    int n = 0;
    for (; n < nbox && n < kRhsGroup; ++n) {
        int64_t v = 1;
        for (int d = 0; d < 3; ++d) v *= boxes[n].hi[d] - boxes[n].lo[d] + 1;
        cells += v;
        if (n > 0 && cells > kRhsGroupCells) break;
    }
    return n;
}

}  // namespace mfg

extern "C" int mfg_set_face_compaction(int on) {
    if (cudaDeviceSynchronize() != cudaSuccess) return MFG_ERR_CUDA;
    mfg::g_face_split = on != 0;
    return MFG_OK;
}
