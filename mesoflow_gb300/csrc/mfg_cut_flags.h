// State of a stored cut-cell entry (mfg_ib.cu) as a flag word, and how a grown
// cell's volume fraction and the end of a pass change it.
//
// The entry keeps a copy of the volume fraction.  A value that moved within its
// kind (gas, cut, solid) goes into the copy, and the weights must be computed
// again (MOVED); a cell of another kind leaves the copy as it is, and the entry
// cannot be applied in this pass (OTHER).  So the kinds of the copy stay those the
// entry was built for, a geometry that comes back finds its entry again, and values
// that moved meanwhile are still owed to the weights: a pass with OTHER leaves
// MOVED behind.  LEFT marks an entry that could not be applied in its last pass,
// for cutcache_sweep to drop.
#pragma once
#include "mfg_fixed.cuh"

namespace mfg {

constexpr unsigned VF_MOVED = 1u, VF_OTHER = 2u, VF_LEFT = 4u;

MFG_HD int vf_kind(double v) { return v == 1.0 ? 2 : (v > 0.0 && v < 1.0) ? 1 : 0; }

// Flag bits of one cell: value v against the copy, which takes it where the kind is the same.
MFG_HD unsigned vf_change(double v, double* copy) {
    const double old = *copy;
    if (bits_of(v) == bits_of(old)) return 0u;
    if (vf_kind(v) != vf_kind(old)) return VF_OTHER;
    *copy = v;
    return VF_MOVED;
}

// What a pass does with the entry.
MFG_HD bool vf_apply(unsigned flag) { return !(flag & VF_OTHER); }
MFG_HD bool vf_refresh(unsigned flag) { return (flag & (VF_MOVED | VF_OTHER)) == VF_MOVED; }
// The flag when the pass is over.
MFG_HD unsigned vf_after(unsigned flag) { return (flag & VF_OTHER) ? VF_MOVED | VF_LEFT : 0u; }

}  // namespace mfg
