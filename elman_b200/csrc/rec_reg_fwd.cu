// Instantiations of the register-resident recurrence kernel, forward (a file per direction: they
// compile in parallel).
#include "rec_reg_table.cuh"

namespace elman {

RecRegKernel rec_reg_fwd_kernel(int mt, int kb, int nt) { return rr::pick<false>(mt, kb, nt); }

}  // namespace elman
