// Instantiations of the register-resident low-rank recurrence with the rank vector in two parts, forward.
#include "lowrank_reg_table.cuh"

namespace elman {

LowRankRegKernel lowrank_split_fwd_kernel(int kb1, int kb2, int mt, int nt) {
  return rr::pick_lowrank<false, true>(kb1, kb2, mt, nt);
}

}  // namespace elman
