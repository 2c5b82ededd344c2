// Run-time (KB1, KB2, MT, NT) -> instantiation of lowrank_reg_kernel; null for others.
#pragma once

#include "lowrank_reg.cuh"

namespace elman {

typedef void (*LowRankRegKernel)(const LowRankRegParams);
// KB1 even (widths in steps of 512), KB2 1 or 2 (rank up to 512), MT 1, 2, 4 or 6, NT 1 or 2
LowRankRegKernel lowrank_reg_fwd_kernel(int kb1, int kb2, int mt, int nt);
LowRankRegKernel lowrank_reg_bwd_kernel(int kb1, int kb2, int mt, int nt);
// the same with the rank vector in two parts
LowRankRegKernel lowrank_split_fwd_kernel(int kb1, int kb2, int mt, int nt);
LowRankRegKernel lowrank_split_bwd_kernel(int kb1, int kb2, int mt, int nt);

namespace rr {

template <bool BWD, bool SPLIT, int KB1, int KB2, int MT>
LowRankRegKernel lr_by_nt(int nt) {
  return nt == 1 ? lowrank_reg_kernel<BWD, KB1, KB2, MT, 1, SPLIT>
         : nt == 2 ? lowrank_reg_kernel<BWD, KB1, KB2, MT, 2, SPLIT> : nullptr;
}
template <bool BWD, bool SPLIT, int KB1, int KB2>
LowRankRegKernel lr_by_mt(int mt, int nt) {
  switch (mt) {
    case 1: return lr_by_nt<BWD, SPLIT, KB1, KB2, 1>(nt);
    case 2: return lr_by_nt<BWD, SPLIT, KB1, KB2, 2>(nt);
    case 4: return lr_by_nt<BWD, SPLIT, KB1, KB2, 4>(nt);
    case 6: return lr_by_nt<BWD, SPLIT, KB1, KB2, 6>(nt);
  }
  return nullptr;
}
template <bool BWD, bool SPLIT, int KB1>
LowRankRegKernel lr_by_kb2(int kb2, int mt, int nt) {
  return kb2 == 1 ? lr_by_mt<BWD, SPLIT, KB1, 1>(mt, nt) : kb2 == 2 ? lr_by_mt<BWD, SPLIT, KB1, 2>(mt, nt) : nullptr;
}
template <bool BWD, bool SPLIT>
LowRankRegKernel pick_lowrank(int kb1, int kb2, int mt, int nt) {
  switch (kb1) {
    case 2: return lr_by_kb2<BWD, SPLIT, 2>(kb2, mt, nt);
    case 4: return lr_by_kb2<BWD, SPLIT, 4>(kb2, mt, nt);
    case 6: return lr_by_kb2<BWD, SPLIT, 6>(kb2, mt, nt);
    case 8: return lr_by_kb2<BWD, SPLIT, 8>(kb2, mt, nt);
  }
  return nullptr;
}

}  // namespace rr
}  // namespace elman
