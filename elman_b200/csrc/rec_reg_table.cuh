// Run-time (MT, KB, NT) -> instantiation of rec_reg_kernel; null outside the register budget.
#pragma once

#include "rec_turns.cuh"

namespace elman {

typedef void (*RecRegKernel)(const RecRegParams);
RecRegKernel rec_reg_fwd_kernel(int mt, int kb, int nt);
RecRegKernel rec_reg_bwd_kernel(int mt, int kb, int nt);

// the same for rec_turns_kernel, with the most rows of W that the registers hold
RecRegKernel rec_turns_fwd_kernel(int kb);
RecRegKernel rec_turns_bwd_kernel(int kb);

namespace rr {

constexpr int turns_mt(int kb) { return kb <= RR_MAX_W / RR_MAX_MT ? RR_MAX_MT : RR_MAX_W / kb; }

template <bool BWD>
RecRegKernel pick_turns(int kb) {
  switch (kb) {
    case 1: return rec_turns_kernel<BWD, turns_mt(1), 1>;
    case 2: return rec_turns_kernel<BWD, turns_mt(2), 2>;
    case 3: return rec_turns_kernel<BWD, turns_mt(3), 3>;
    case 4: return rec_turns_kernel<BWD, turns_mt(4), 4>;
    case 5: return rec_turns_kernel<BWD, turns_mt(5), 5>;
    case 6: return rec_turns_kernel<BWD, turns_mt(6), 6>;
    case 7: return rec_turns_kernel<BWD, turns_mt(7), 7>;
    case 8: return rec_turns_kernel<BWD, turns_mt(8), 8>;
  }
  return nullptr;
}

template <bool BWD, int MT, int KB, int NT>
RecRegKernel one() {
  if constexpr (MT * KB <= RR_MAX_W) return rec_reg_kernel<BWD, MT, KB, NT>;
  else return nullptr;
}
template <bool BWD, int MT, int KB>
RecRegKernel by_nt(int nt) {
  return nt == 1 ? one<BWD, MT, KB, 1>() : nt == 2 ? one<BWD, MT, KB, 2>() : nullptr;
}
template <bool BWD, int MT>
RecRegKernel by_kb(int kb, int nt) {
  switch (kb) {
    case 1: return by_nt<BWD, MT, 1>(nt);
    case 2: return by_nt<BWD, MT, 2>(nt);
    case 3: return by_nt<BWD, MT, 3>(nt);
    case 4: return by_nt<BWD, MT, 4>(nt);
    case 5: return by_nt<BWD, MT, 5>(nt);
    case 6: return by_nt<BWD, MT, 6>(nt);
    case 7: return by_nt<BWD, MT, 7>(nt);
    case 8: return by_nt<BWD, MT, 8>(nt);
  }
  return nullptr;
}
template <bool BWD>
RecRegKernel pick(int mt, int kb, int nt) {
  switch (mt) {
    case 1: return by_kb<BWD, 1>(kb, nt);
    case 2: return by_kb<BWD, 2>(kb, nt);
    case 3: return by_kb<BWD, 3>(kb, nt);
    case 4: return by_kb<BWD, 4>(kb, nt);
  }
  return nullptr;
}

}  // namespace rr
}  // namespace elman
