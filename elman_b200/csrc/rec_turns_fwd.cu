// Instantiations of the turn-taking recurrence kernel, forward.
#include "rec_reg_table.cuh"

namespace elman {

RecRegKernel rec_turns_fwd_kernel(int kb) { return rr::pick_turns<false>(kb); }

}  // namespace elman
