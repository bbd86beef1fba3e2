// Step bookends and chemistry: reaction source, SSP-RK3 chemistry sub-step,
// primitive refresh, species clipping, residual norms and the CFL estimate.
#include "mfg_step_body.cuh"

namespace mfg {
namespace {

constexpr int TPB = 256;

template <int NS>
__global__ void chem_source_kernel(Valid v, Fab S, Fab D) {
    chem_source_body<NS>(v, S, D, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
// Boxes of one launch of the chemistry sub-step, primitive refresh and clipping
// (blockIdx.y).
constexpr int LOCAL_GROUP = 8;
struct LocalGroup {
    Valid v[LOCAL_GROUP];
    Fab so[LOCAL_GROUP], sn[LOCAL_GROUP];
};
template <int NS>
__global__ void chem_substep_kernel(const __grid_constant__ LocalGroup g, double dt, int ncomp) {
    const int q = blockIdx.y;
    chem_substep_body<NS>(g.v[q], g.so[q], g.sn[q], dt, ncomp, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
template <int NS>
__global__ void prims_kernel(const __grid_constant__ LocalGroup g) {
    prims_body<NS>(g.v[blockIdx.y], g.sn[blockIdx.y], (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}
template <int NS>
__global__ void chem_rk2_kernel(Valid v, Fab So, Fab Sn, double dt, int ncomp) {
    chem_rk2_body<NS>(v, So, Sn, dt, ncomp, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

template <int NS>
__global__ void inertgas_kernel(Valid v, Fab S) {
    inertgas_body<NS>(v, S, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

template <int NS>
__global__ void vars_after_chem_kernel(Valid v, Fab S, int bg) {
    vars_after_chem_body<NS>(v, S, bg, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void clip_kernel(const __grid_constant__ LocalGroup g, int nspec) {
    clip_body(g.v[blockIdx.y], g.sn[blockIdx.y], nspec, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

// Block partial sums of ((s_new - s_old)/dt [* vfrac_old])^2 per component;
// warp-shuffle reduction inside the block, partials in block order.
__global__ void resnorm_kernel(Valid v, Fab Sn, Fab So, double a, double b, double* partial, int nblk) {
    const int n = blockIdx.y;
    double acc = 0.0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < v.n; t += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        cell_of(v, t, i, j, k);
        // LinComb then Multiply, rounded as the reference (no contraction)
        double d = add(mul(a, Sn(i, j, k, n)), mul(b, So(i, j, k, n)));
        if (n < VFRAC) d = mul(d, So(i, j, k, VFRAC));
        acc += d * d;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    __shared__ double ws[TPB / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double x = (threadIdx.x < TPB / 32) ? ws[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (threadIdx.x == 0) partial[(int64_t)n * nblk + blockIdx.x] = x;
    }
}

// The bookends of a box after the RK3 stages in one pass (post_cell: phi_old
// <- phi_new and the chemistry sub-step when chem, primitive refresh, species
// clipping when clip) and, when partial != nullptr, the block partial sums of
// the residual norms ((s_new - s_old)/dt, flow components scaled by the old
// volume fraction).  Each thread keeps one running sum per component in
// registers (with the chemistry sub-step, only the components the bookends
// change can be non-zero); the block then sums them by warp shuffles and one
// warp adds the warps' sums in a fixed order, so the partials are
// deterministic.
//
// One launch serves a group of boxes (blockIdx.y): a small box alone leaves
// most of the GPU idle.  Every box keeps its own partials, reduced over its own
// blocks, and the final sum adds the boxes in order: the norms' bits do not
// depend on the grouping.
constexpr int PTPB = 128;
constexpr int PARTIALS = 1024;  // per box and component

struct PostGroup {
    Valid v[kRhsGroup];
    Fab so[kRhsGroup], sn[kRhsGroup];
    int nblk[kRhsGroup];
};

template <int NS, int CHEM, bool NORMS>
__global__ void __launch_bounds__(PTPB) post_step_kernel(const __grid_constant__ PostGroup g, double dt, int clip,
                                                         double a, double b, double* partial) {
    constexpr int NM = NFLO + NS;
    const int N = NFLO + c_P.nspec;
    const int q = blockIdx.y, nblk = g.nblk[q];
    if (blockIdx.x >= nblk) return;
    const Valid& v = g.v[q];
    const Fab &So = g.so[q], &Sn = g.sn[q];
    double acc[NM];
#pragma unroll
    for (int n = 0; n < NM; ++n) acc[n] = 0.0;
    bool nonfinite = false;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < v.n; t += (int64_t)nblk * blockDim.x) {
        int i, j, k;
        cell_of(v, t, i, j, k);
        post_cell<NS, CHEM, NORMS>(So, Sn, i, j, k, dt, clip != 0, a, b, acc, nonfinite);
    }
    if (!NORMS) return;
    const int any_nonfinite = __syncthreads_or(nonfinite ? 1 : 0);
    __shared__ double ws[PTPB / 32][NM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int n = 0; n < NM; ++n) {
        if (CHEM != 0 && !(n >= DENS && n <= TEMP) && n < NFLO) continue;  // zero in every cell
        double x = acc[n];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) ws[warp][n] = x;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        const int n = threadIdx.x;
        double x;
        if (CHEM != 0 && !(n >= DENS && n <= TEMP) && n < NFLO) {
            x = any_nonfinite ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
        } else {
            x = 0.0;
            for (int w = 0; w < PTPB / 32; ++w) x += ws[w][n];
        }
        partial[((int64_t)q * N + n) * PARTIALS + blockIdx.x] = x;
    }
}

// Fixed-order final sum of the block partials of one box, accumulated into acc[n].
__global__ void resnorm_final_kernel(const double* partial, int nblk, double* acc) {
    const int n = blockIdx.x;
    double x = 0.0;
    for (int b = threadIdx.x; b < nblk; b += 32) x += partial[(int64_t)n * nblk + b];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (threadIdx.x == 0) acc[n] += x;
}
// The same for a group's boxes, box after box.
__global__ void post_final_kernel(const __grid_constant__ PostGroup g, int nbox, const double* partial, double* acc) {
    const int n = blockIdx.x, N = gridDim.x;
    double sum = acc[n];
    for (int q = 0; q < nbox; ++q) {
        double x = 0.0;
        for (int b = threadIdx.x; b < g.nblk[q]; b += 32) x += partial[((int64_t)q * N + n) * PARTIALS + b];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        sum += x;  // lane 0's is the box's sum
    }
    if (threadIdx.x == 0) acc[n] = sum;
}

// max wavespeed and max species diffusivity (Source/mflo_timestep.cpp:83-133)
// over a group of boxes (blockIdx.y)
constexpr int STEP_GROUP = 16;
struct StepGroup {
    Valid v[STEP_GROUP];
    Fab s[STEP_GROUP];
};
template <int NS>
__global__ void timestep_kernel(const __grid_constant__ StepGroup g, double* acc2) {
    const Valid& v = g.v[blockIdx.y];
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t - threadIdx.x >= v.n) return;  // whole block past this box
    double ws = 0.0, md = 0.0;
    if (t < v.n) {
        int i, j, k;
        cell_of(v, t, i, j, k);
        timestep_cell<NS>(g.s[blockIdx.y], i, j, k, ws, md);
    }
    warp_max_nonneg(acc2, ws);
    warp_max_nonneg(acc2 + 1, md);
}

// Contiguous copies of several arrays in one launch (blockIdx.y = array), four
// loads in flight per thread.
constexpr int COPY_GROUP = 32;
struct CopyList {
    const double* src[COPY_GROUP];
    double* dst[COPY_GROUP];
    int64_t n[COPY_GROUP];
};
__global__ void __launch_bounds__(TPB) copy_list_kernel(const __grid_constant__ CopyList g) {
    const double* __restrict__ src = g.src[blockIdx.y];
    double* __restrict__ dst = g.dst[blockIdx.y];
    const int64_t n = g.n[blockIdx.y], base = (int64_t)blockIdx.x * (4 * TPB) + threadIdx.x;
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = (base + u * TPB < n) ? src[base + u * TPB] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (base + u * TPB < n) dst[base + u * TPB] = v[u];
}

// dst = (copy_first ? base : dst) + a*src over the valid box, all components.
__global__ void axpy_kernel(Valid v, Fab dst, Fab src, double a, int copy_first, Fab base, int ncomp) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int n = blockIdx.y;
    if (t >= v.n || n >= ncomp) return;
    int i, j, k;
    cell_of(v, t, i, j, k);
    double x = copy_first ? base(i, j, k, n) : dst(i, j, k, n);
    if (src.p) x = add(x, mul(a, src(i, j, k, n)));
    dst(i, j, k, n) = x;
}

inline unsigned nblocks(int64_t n) { return (unsigned)((n + TPB - 1) / TPB); }

}  // namespace

cudaError_t launch_chem_source(const mfg_box& b, cudaStream_t st) {
    Valid v = valid_of(b);
    Fab S = make_fab(b.s_new), D = make_fab(b.dsdt);
    const int ns = c_host_params().nspec;
    ProfScope ps(K_CHEM, st);
    if (ns <= 1) chem_source_kernel<1><<<nblocks(v.n), TPB, 0, st>>>(v, S, D);
    else if (ns <= 2) chem_source_kernel<2><<<nblocks(v.n), TPB, 0, st>>>(v, S, D);
    else if (ns <= 4) chem_source_kernel<4><<<nblocks(v.n), TPB, 0, st>>>(v, S, D);
    else if (ns <= 8) chem_source_kernel<8><<<nblocks(v.n), TPB, 0, st>>>(v, S, D);
    else chem_source_kernel<16><<<nblocks(v.n), TPB, 0, st>>>(v, S, D);
    return cudaGetLastError();
}

// Calls f(group, grid) for the boxes, LOCAL_GROUP at a time.
template <class F>
static cudaError_t for_local_groups(const mfg_box* boxes, int nbox, F&& f) {
    for (int b = 0; b < nbox; b += LOCAL_GROUP) {
        const int n = std::min(LOCAL_GROUP, nbox - b);
        LocalGroup g;
        int64_t most = 0;
        for (int q = 0; q < LOCAL_GROUP; ++q) {
            const mfg_box& x = boxes[b + (q < n ? q : 0)];
            g.v[q] = valid_of(x);
            g.so[q] = make_fab(x.s_old);
            g.sn[q] = make_fab(x.s_new);
            most = std::max(most, g.v[q].n);
        }
        f(g, dim3(nblocks(most), n));
    }
    return cudaGetLastError();
}

cudaError_t launch_chem_substep(const mfg_box* boxes, int nbox, double dt, cudaStream_t st) {
    const int ns = c_host_params().nspec, nc = NFLO + ns;
    return for_local_groups(boxes, nbox, [&](const LocalGroup& g, dim3 grid) {
        ProfScope ps(K_CHEM, st);
        if (ns <= 1) chem_substep_kernel<1><<<grid, TPB, 0, st>>>(g, dt, nc);
        else if (ns <= 2) chem_substep_kernel<2><<<grid, TPB, 0, st>>>(g, dt, nc);
        else if (ns <= 4) chem_substep_kernel<4><<<grid, TPB, 0, st>>>(g, dt, nc);
        else if (ns <= 8) chem_substep_kernel<8><<<grid, TPB, 0, st>>>(g, dt, nc);
        else if (ns <= 12) chem_substep_kernel<12><<<grid, TPB, 0, st>>>(g, dt, nc);
        else chem_substep_kernel<16><<<grid, TPB, 0, st>>>(g, dt, nc);
    });
}

cudaError_t launch_update_prims(const mfg_box* boxes, int nbox, cudaStream_t st) {
    const int ns = c_host_params().nspec;
    return for_local_groups(boxes, nbox, [&](const LocalGroup& g, dim3 grid) {
        ProfScope ps(K_PRIMS, st);
        if (ns <= 1) prims_kernel<1><<<grid, TPB, 0, st>>>(g);
        else if (ns <= 2) prims_kernel<2><<<grid, TPB, 0, st>>>(g);
        else if (ns <= 4) prims_kernel<4><<<grid, TPB, 0, st>>>(g);
        else if (ns <= 8) prims_kernel<8><<<grid, TPB, 0, st>>>(g);
        else prims_kernel<16><<<grid, TPB, 0, st>>>(g);
    });
}

// Split-chemistry pieces (Source/mflo_splitchem.cpp): kind 0 Advance_chemistry,
// 1 store_inertgas_conc, 2 update_vars_after_chemsolve (bg = using_bg_inertgas).
cudaError_t launch_split_chem(const mfg_box& b, int kind, double dt, int bg, cudaStream_t st) {
    Valid v = valid_of(b);
    Fab So = make_fab(b.s_old), Sn = make_fab(b.s_new);
    const int ns = c_host_params().nspec, nc = NFLO + ns;
    const unsigned g = nblocks(v.n);
    ProfScope ps(K_CHEM, st);
#define MFG_SPLIT(NSB)                                                                  \
    if (kind == 0) chem_rk2_kernel<NSB><<<g, TPB, 0, st>>>(v, So, Sn, dt, nc);         \
    else if (kind == 1) inertgas_kernel<NSB><<<g, TPB, 0, st>>>(v, Sn);                \
    else vars_after_chem_kernel<NSB><<<g, TPB, 0, st>>>(v, Sn, bg);
    if (ns <= 1) { MFG_SPLIT(1) }
    else if (ns <= 2) { MFG_SPLIT(2) }
    else if (ns <= 4) { MFG_SPLIT(4) }
    else if (ns <= 8) { MFG_SPLIT(8) }
    else { MFG_SPLIT(16) }
#undef MFG_SPLIT
    return cudaGetLastError();
}

cudaError_t launch_clip_species(const mfg_box* boxes, int nbox, cudaStream_t st) {
    return for_local_groups(boxes, nbox, [&](const LocalGroup& g, dim3 grid) {
        ProfScope ps(K_CLIP, st);
        clip_kernel<<<grid, TPB, 0, st>>>(g, c_host_params().nspec);
    });
}

// partial: scratch of (ncomp * 1024) doubles; acc: ncomp doubles (device).
cudaError_t launch_resnorm_box(const mfg_box& b, double dt, double* partial, double* acc, cudaStream_t st) {
    Valid v = valid_of(b);
    const int nc = NFLO + c_host_params().nspec;
    // 16 cells per thread: blocks of one cell per thread were dominated by their fixed cost
    int nblk = (int)std::max<int64_t>(1, std::min<int64_t>(1024, (v.n + 16 * TPB - 1) / (16 * TPB)));
    dim3 g(nblk, nc);
    ProfScope ps(K_RESNORM, st, 2);
    resnorm_kernel<<<g, TPB, 0, st>>>(v, make_fab(b.s_new), make_fab(b.s_old), 1.0 / dt, -1.0 / dt, partial, nblk);
    resnorm_final_kernel<<<nc, 32, 0, st>>>(partial, nblk, acc);
    return cudaGetLastError();
}

// The bookends of n <= kRhsGroup boxes.  partial: scratch of (n * ncomp * 1024)
// doubles, acc: ncomp doubles (device), or both null (no residual norms).
cudaError_t launch_post_step(const mfg_box* boxes, int n, double dt, bool chem, bool clip, double* partial, double* acc,
                             cudaStream_t st) {
    const int ns = c_host_params().nspec, nc = NFLO + ns;
    // one cell per thread up to one wave of blocks (4 of 128 threads resident
    // per SM at the kernel's ~115 registers), then a grid-stride loop: every
    // thread ends with warp sums of its norm terms, so fewer threads with
    // more cells each spend less of the FP64 pipe on them (3.37 -> 3.10 ms per
    // 256^3 step against 1024 blocks); at most 1024 (the partials' scratch)
    static int wave = 0;
    if (!wave) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        wave = std::max(1, std::min(PARTIALS, 4 * sms));
    }
    PostGroup g;
    int most = 1;
    for (int q = 0; q < kRhsGroup; ++q) {
        const mfg_box& b = boxes[q < n ? q : 0];
        g.v[q] = valid_of(b);
        g.so[q] = make_fab(b.s_old);
        g.sn[q] = make_fab(b.s_new);
        g.nblk[q] = (int)std::max<int64_t>(1, std::min<int64_t>(wave, (g.v[q].n + PTPB - 1) / PTPB));
        if (q < n) most = std::max(most, g.nblk[q]);
    }
    const dim3 grid(most, n);
    const double a = 1.0 / dt, bb = -1.0 / dt;
    const DevParams& P = c_host_params();
    // the sub-step of a zero source (no reactions, explicit integrator) is s + 0
    const int kind = !chem ? 0 : (P.chem_kind == 0 && (!P.chem_on || P.nreact == 0)) ? 1 : 2;
    ProfScope ps(K_POST, st, partial ? 2 : 1);
#define MFG_POST_K(NSB, K)                                                                    \
    if (partial)                                                                              \
        post_step_kernel<NSB, K, true><<<grid, PTPB, 0, st>>>(g, dt, clip, a, bb, partial);   \
    else                                                                                      \
        post_step_kernel<NSB, K, false><<<grid, PTPB, 0, st>>>(g, dt, clip, a, bb, partial)
#define MFG_POST(NSB)                     \
    if (kind == 0) MFG_POST_K(NSB, 0);    \
    else if (kind == 1) MFG_POST_K(NSB, 1); \
    else MFG_POST_K(NSB, 2);
    if (ns <= 1) { MFG_POST(1) }
    else if (ns <= 2) { MFG_POST(2) }
    else if (ns <= 4) { MFG_POST(4) }
    else if (ns <= 8) { MFG_POST(8) }
    else if (ns <= 12 && kind == 2) { MFG_POST_K(12, 2); }  // the reactions' arrays for 16 species spill
    else { MFG_POST(16) }
#undef MFG_POST
#undef MFG_POST_K
    if (partial) post_final_kernel<<<nc, 32, 0, st>>>(g, n, partial, acc);
    return cudaGetLastError();
}

cudaError_t launch_timestep(const mfg_box* boxes, int nbox, double* acc2, cudaStream_t st) {
    const int ns = c_host_params().nspec;
    for (int b = 0; b < nbox; b += STEP_GROUP) {
        const int n = std::min(STEP_GROUP, nbox - b);
        StepGroup g;
        int64_t most = 0;
        for (int q = 0; q < STEP_GROUP; ++q) {
            const mfg_box& x = boxes[b + (q < n ? q : 0)];
            g.v[q] = valid_of(x);
            g.s[q] = make_fab(x.s_new);
            most = std::max(most, g.v[q].n);
        }
        const dim3 grid(nblocks(most), n);
        ProfScope ps(K_TIMESTEP, st);
        if (ns <= 1) timestep_kernel<1><<<grid, TPB, 0, st>>>(g, acc2);
        else if (ns <= 2) timestep_kernel<2><<<grid, TPB, 0, st>>>(g, acc2);
        else if (ns <= 4) timestep_kernel<4><<<grid, TPB, 0, st>>>(g, acc2);
        else if (ns <= 8) timestep_kernel<8><<<grid, TPB, 0, st>>>(g, acc2);
        else timestep_kernel<16><<<grid, TPB, 0, st>>>(g, acc2);
    }
    return cudaGetLastError();
}

// Whether f holds exactly the valid box, components one after the other,
// with no padding (then a copy of it is one contiguous block).
static bool dense_over(const Fab& f, const mfg_box& b) {
    const int64_t l0 = b.hi[0] - b.lo[0] + 1, l1 = b.hi[1] - b.lo[1] + 1, l2 = b.hi[2] - b.lo[2] + 1;
    return f.p && f.b0 == b.lo[0] && f.b1 == b.lo[1] && f.b2 == b.lo[2] && f.js == l0 && f.ks == l0 * l1 &&
           f.ns == l0 * l1 * l2;
}

cudaError_t launch_axpy_valid(const mfg_box& b, const Fab& dst, const Fab& src, double a, bool copy_first,
                              const Fab& base, int ncomp, cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const cudaError_t ce = cudaStreamIsCapturing(st, &cs);
    if (ce != cudaSuccess) return ce;
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    if (copy_first && !src.p && !capturing && dense_over(dst, b) && dense_over(base, b)) {
        // a plain copy of two dense arrays (phi_old <- phi_new): one block
        // copy at the copy bandwidth instead of a kernel per (cell, component)
        // (graphs keep the kernel: their conditional bodies take kernels);
        // arrays that overlap without being the same one take the kernel, whose
        // per-cell copy is defined for them
        const size_t bytes = (size_t)ncomp * dst.ns * sizeof(double);
        if (dst.p == base.p) {
            ProfScope ps(K_COPY, st, 0);
            return cudaSuccess;
        }
        const char *d0 = reinterpret_cast<const char*>(dst.p), *b0 = reinterpret_cast<const char*>(base.p);
        if (d0 + bytes <= b0 || b0 + bytes <= d0) {
            ProfScope ps(K_COPY, st, 0);
            return cudaMemcpyAsync(dst.p, base.p, bytes, cudaMemcpyDeviceToDevice, st);
        }
    }
    Valid v = valid_of(b);
    dim3 g(nblocks(v.n), ncomp);
    ProfScope ps(K_COPY, st);
    axpy_kernel<<<g, TPB, 0, st>>>(v, dst, src, a, copy_first ? 1 : 0, base, ncomp);
    return cudaGetLastError();
}

// phi_old <- phi_new of every box (not for stream capture): dense arrays, in
// the same layout and apart from each other, by copy_list_kernel, the others
// box by box.
cudaError_t launch_copy_old(const mfg_box* boxes, int nbox, int ncomp, cudaStream_t st) {
    Fab none;
    memset(&none, 0, sizeof(none));
    CopyList g;
    int n = 0;
    int64_t most = 0;
    auto flush = [&]() {
        if (!n) return;
        ProfScope ps(K_COPY, st);
        copy_list_kernel<<<dim3((unsigned)((most + 4 * TPB - 1) / (4 * TPB)), n), TPB, 0, st>>>(g);
        n = 0;
        most = 0;
    };
    for (int b = 0; b < nbox; ++b) {
        const Fab d = make_fab(boxes[b].s_old), s = make_fab(boxes[b].s_new);
        const int64_t cnt = (int64_t)ncomp * d.ns;
        const bool apart = d.p + cnt <= s.p || s.p + cnt <= d.p;
        if (d.p == s.p && dense_over(d, boxes[b]) && dense_over(s, boxes[b])) continue;
        if (!apart || !dense_over(d, boxes[b]) || !dense_over(s, boxes[b])) {
            flush();
            const cudaError_t e = launch_axpy_valid(boxes[b], d, none, 0.0, true, s, ncomp, st);
            if (e != cudaSuccess) return e;
            continue;
        }
        g.src[n] = s.p;
        g.dst[n] = d.p;
        g.n[n++] = cnt;
        most = std::max(most, cnt);
        if (n == COPY_GROUP) flush();
    }
    flush();
    return cudaGetLastError();
}

}  // namespace mfg
