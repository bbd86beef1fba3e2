// Launches of the flow right-hand side and fused RK3 stage update over a group
// of boxes: every phase is one launch for all boxes of the group (blockIdx.z)
// and, for the face and flux passes, all three directions.
//
// A box of 16 to 32 cells per side gives a launch 10 to 250 thousand threads of
// the 300 thousand that fill the GPU, and 8 launches per box and stage cost
// more than their work; up to kRhsGroup boxes together (rhs_group_count) share
// a launch, each with its own scratch.  The boxes travel as a kernel parameter:
// no table in device memory to build, upload or keep.  G = 1 is the same for a
// single box with a parameter of one box's size.  Boxes of different sizes
// share a grid of the largest one's blocks; blocks past a box's items exit.
#pragma once
#include <algorithm>

#include "mfg_rhs_body.cuh"

namespace mfg {
namespace {

constexpr int TPB = 256;

template <int G>
struct RhsGroup {
    RhsBox b[G];
};

template <int NS, int G>
__global__ void __launch_bounds__(TPB) prim_kernel(const __grid_constant__ RhsGroup<G> g) {
    const Fp fp;
    prim_body<NS>(fp, g.b[G == 1 ? 0 : blockIdx.z], (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
// HIGH: orders 4 and 5 (face scalars), else orders 1 and 2 in one pass.
// Without the AUSM+-up branch the face scalars need 76 registers, so the two
// are compiled apart: with one kernel for both, a block of 256 threads at 132
// registers was alone on its SM (64^3 box, three directions: 155 -> 86 us).
template <int NS, int G, bool HIGH>
__global__ void __launch_bounds__(TPB) face_kernel(const __grid_constant__ RhsGroup<G> g) {
    const Fp fp;
    const int d = blockIdx.y;
    face_body<NS, HIGH>(fp, g.b[G == 1 ? 0 : blockIdx.z], d, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
// Orders 1 and 2 with Navier-Stokes terms: the inactive faces (solid side,
// conduction and diffusion only) of all three directions are written here
// (blockIdx.y = direction) and the active ones listed per direction (one
// atomic per warp), so that face_list_kernel runs the flux branch of all
// three directions in one launch with every lane of a warp busy (blocks past
// a direction's count exit at once).  Same
// per-face arithmetic: bitwise the results of face_kernel.
__device__ __forceinline__ int64_t face_list_off(const RhsBox& B, int d) {
    int64_t o = 0;
    for (int e = 0; e < d; ++e) o += face_count(B, e);
    return o;
}
template <int G>
__global__ void fcount_reset_kernel(const __grid_constant__ RhsGroup<G> g, int n) {
    const int b = threadIdx.x / 3;
    if (b < n) g.b[b].fcount[threadIdx.x % 3] = 0;
}
template <int NS, int G>
__global__ void __launch_bounds__(TPB) face_split_kernel(const __grid_constant__ RhsGroup<G> g) {
    const Fp fp;
    const RhsBox& B = g.b[G == 1 ? 0 : blockIdx.z];
    const int d = blockIdx.y;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool act = false;
    int lo[3] = {B.lo[0], B.lo[1], B.lo[2]}, len[3];
    for (int e = 0; e < 3; ++e) len[e] = B.hi[e] - B.lo[e] + 1 + (e == d);
    if (t < (int64_t)len[0] * len[1] * len[2]) {
        const Idx3 f = delinear(t, lo, len);  // once for the test and the body
        act = face_active(fp, B, d, f);
        if (!act) face_body_at<NS, false, true>(fp, B, d, f);
    }
    const unsigned m = __ballot_sync(0xffffffffu, act);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    unsigned base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(B.fcount + d, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    if (act) B.flist[face_list_off(B, d) + base + __popc(m & ((1u << lane) - 1u))] = (int)t;
}
// The direction is the block's (blockIdx.y), uniform as in face_kernel.
// 128-thread blocks.  One or two species: 5 per SM (96 registers), 1% faster
// than 4; more species need 128 registers (5 per SM spill: 8% slower with ten).
constexpr int LIST_TPB = 128;
template <int NS, int G>
__global__ void __launch_bounds__(LIST_TPB, NS <= 2 ? 5 : 4) face_list_kernel(const __grid_constant__ RhsGroup<G> g) {
    const RhsBox& B = g.b[G == 1 ? 0 : blockIdx.z];
    const int d = blockIdx.y;
    const unsigned w = blockIdx.x * blockDim.x + threadIdx.x;
    const Fp fp;
    if (w < B.fcount[d]) face_body<NS, false, true>(fp, B, d, B.flist[face_list_off(B, d) + w]);
}
// Direction and box of the flux launches: blockIdx.z = 3 box + direction.
template <int G>
__global__ void __launch_bounds__(TPB) flux4_kernel(const __grid_constant__ RhsGroup<G> g) {
    const Fp fp;
    flux4_body(fp, g.b[G == 1 ? 0 : blockIdx.z / 3], blockIdx.z % 3, blockIdx.y,
               (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
template <int G>
__global__ void __launch_bounds__(TPB) flux_kernel(const __grid_constant__ RhsGroup<G> g) {
    flux_body(g.b[G == 1 ? 0 : blockIdx.z / 3], blockIdx.z % 3, blockIdx.y,
                    (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
constexpr int SWEEP_TPB = 128;
// Four blocks per SM (128 registers): 16 warps keep the FP64 and integer pipes
// busier than 12 (168 registers): 24.6 against 25.7 ms per 128^3 Taylor-Green
// step when that was measured, 16 ms with the operations cut since.
template <int G>
__global__ void __launch_bounds__(SWEEP_TPB, 4) flux5_sweep_kernel(const __grid_constant__ RhsGroup<G> g, int seg) {
    const Fp fp;
    flux5_sweep_body(fp, g.b[G == 1 ? 0 : blockIdx.z / 3], blockIdx.z % 3, blockIdx.y,
                     (int64_t)blockIdx.x * blockDim.x + threadIdx.x, seg);
}
template <int G>
__global__ void __launch_bounds__(SWEEP_TPB, 4) flux5_face_kernel(const __grid_constant__ RhsGroup<G> g) {
    const Fp fp;
    flux5_face_body(fp, g.b[G == 1 ? 0 : blockIdx.z / 3], blockIdx.z % 3, blockIdx.y,
                    (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
// The column segments of a launch must fill the GPU: segments of 32, 16, 8 or 4
// faces (longer ones share more per-cell work), else the per-face form of the
// same arithmetic, which does about twice the work per face.  A 16^3 box with
// 13 advected components takes the per-face form: 58 us per right-hand side (50
// since), against 67 and 84 with half and a quarter of this bound.
constexpr int64_t SWEEP_MIN_THREADS = 152 * 2 * SWEEP_TPB * 2;
template <int G>
__global__ void __launch_bounds__(TPB) update_kernel(const __grid_constant__ RhsGroup<G> g, int stage, double dt) {
    const Fp fp;
    update_body(fp, g.b[G == 1 ? 0 : blockIdx.z], stage, dt, blockIdx.y,
                (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

inline unsigned blocks_for(int64_t n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }

template <int NS, int G>
cudaError_t launch_group_ns(const RhsGroup<G>& g, int n, int stage, double dt, bool fast, bool split_on,
                            cudaStream_t st) {
    const DevParams& P = c_host_params();
    const int C = NCONS + P.nspec, N = NFLO + P.nspec;
    int64_t ng = 0, nv = 0, nf = 0;  // largest box's grown cells, valid cells, faces of a direction
    for (int b = 0; b < n; ++b) {
        ng = std::max(ng, prim_items(g.b[b]));
        nv = std::max(nv, cell_items(g.b[b]));
        for (int d = 0; d < 3; ++d) nf = std::max(nf, face_items(g.b[b], d));
    }
    const int ord = P.order_hyp;
    const bool high = ord == 4 || ord == 5;
    if (high) {
        ProfScope ps(K_PRIM, st);
        prim_kernel<NS, G><<<dim3(blocks_for(ng), 1, n), TPB, 0, st>>>(g);
    }
    if (split_on && P.do_ns && !high) {
        ProfScope ps(K_FACE, st, 3);
        fcount_reset_kernel<G><<<1, 3 * G, 0, st>>>(g, n);
        face_split_kernel<NS, G><<<dim3(blocks_for(nf), 3, n), TPB, 0, st>>>(g);
        face_list_kernel<NS, G><<<dim3(blocks_for(nf, LIST_TPB), 3, n), LIST_TPB, 0, st>>>(g);
    } else {
        ProfScope ps(K_FACE, st);
        const dim3 gf(blocks_for(nf), 3, n);
        if (high)
            face_kernel<NS, G, true><<<gf, TPB, 0, st>>>(g);
        else
            face_kernel<NS, G, false><<<gf, TPB, 0, st>>>(g);
    }
    if (high || !P.do_ns) {  // orders 1, 2 with Navier-Stokes terms: the face kernels wrote the fluxes
        ProfScope ps(K_FLUX, st);
        if (fast && ord == 5 && P.do_ns) {
            int64_t tot = 0;
            int seg = 64;
            do {
                seg /= 2;
                tot = 0;
                for (int b = 0; b < n; ++b)
                    for (int d = 0; d < 3; ++d) tot += sweep_items(g.b[b], d, seg);
            } while (seg > 4 && tot * C < SWEEP_MIN_THREADS);
            if (tot * C >= SWEEP_MIN_THREADS) {
                int64_t most = 0;
                for (int b = 0; b < n; ++b)
                    for (int d = 0; d < 3; ++d) most = std::max(most, sweep_items(g.b[b], d, seg));
                flux5_sweep_kernel<G><<<dim3(blocks_for(most, SWEEP_TPB), C, 3 * n), SWEEP_TPB, 0, st>>>(g, seg);
            } else {
                flux5_face_kernel<G><<<dim3(blocks_for(nf, SWEEP_TPB), C, 3 * n), SWEEP_TPB, 0, st>>>(g);
            }
        } else if (ord == 4 && P.do_ns) {
            flux4_kernel<G><<<dim3(blocks_for(nf), C, 3 * n), TPB, 0, st>>>(g);
        } else {
            flux_kernel<G><<<dim3(blocks_for(nf), C, 3 * n), TPB, 0, st>>>(g);
        }
    }
    ProfScope ps(K_UPDATE, st);
    update_kernel<G><<<dim3(blocks_for(nv), N, n), TPB, 0, st>>>(g, stage, dt);
    return cudaGetLastError();
}

template <int G>
cudaError_t launch_group(const RhsBox* boxes, int n, int stage, double dt, bool fast, bool split_on, cudaStream_t st) {
    RhsGroup<G> g;
    for (int b = 0; b < G; ++b) g.b[b] = boxes[b < n ? b : 0];
    const int ns = c_host_params().nspec;
    if (ns <= 1) return launch_group_ns<1, G>(g, n, stage, dt, fast, split_on, st);
    if (ns <= 2) return launch_group_ns<2, G>(g, n, stage, dt, fast, split_on, st);
    if (ns <= 4) return launch_group_ns<4, G>(g, n, stage, dt, fast, split_on, st);
    if (ns <= 8) return launch_group_ns<8, G>(g, n, stage, dt, fast, split_on, st);
    // 9 to 12 species apart: the face states of 16 spill (AUSM+-up with ten species
    // 383 -> 370 us per right-hand side of 61x47x38 cells; primitives of the 64^3
    // catalyst step 204 -> 172 us)
    if (ns <= 12) return launch_group_ns<12, G>(g, n, stage, dt, fast, split_on, st);
    return launch_group_ns<16, G>(g, n, stage, dt, fast, split_on, st);
}

}  // namespace
}  // namespace mfg
