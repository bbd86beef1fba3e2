// The launches of mfg_rhs_launch.cuh for groups of several boxes (compiled
// beside mfg_rhs.cu's single-box ones).
#include "mfg_rhs_launch.cuh"

namespace mfg {

cudaError_t launch_rhs_group(const RhsBox* boxes, int n, int stage, double dt, bool fast, bool split_on,
                             cudaStream_t st) {
    return launch_group<kRhsGroup>(boxes, n, stage, dt, fast, split_on, st);
}

}  // namespace mfg
