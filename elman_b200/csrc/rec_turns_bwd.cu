// Instantiations of the turn-taking recurrence kernel, backward.
#include "rec_reg_table.cuh"

namespace elman {

RecRegKernel rec_turns_bwd_kernel(int kb) { return rr::pick_turns<true>(kb); }

}  // namespace elman
