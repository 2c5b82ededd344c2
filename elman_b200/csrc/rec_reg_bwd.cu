// Instantiations of the register-resident recurrence kernel, backward (a file per direction: they
// compile in parallel).
#include "rec_reg_table.cuh"

namespace elman {

RecRegKernel rec_reg_bwd_kernel(int mt, int kb, int nt) { return rr::pick<true>(mt, kb, nt); }

}  // namespace elman
