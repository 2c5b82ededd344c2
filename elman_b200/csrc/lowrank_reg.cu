// Plans and launches of the register-resident low-rank recurrence (lowrank_reg.cuh).
#include "lowrank_reg_table.cuh"

namespace elman {

namespace {

struct LowRankRegPlan {
  int kb1, kb2, mt, nt;
  int cpg;          // CTAs per group
  int rows;         // batch rows per launch (a multiple of the group)
  double cost;
  bool ok;
};

// The dense kernel's step model (rec_reg.cu) for two hand-offs.  A batch whose groups do not all
// fit on the device goes through in slices, one launch after the other: sequences are independent.
// Measured, us per step forward / backward, against what ran before:
//
//    B    d    r   before                          this kernel
//   32 1536  270   5.6  6.0  (one cluster, TMEM)   2.37 2.52
//    8 1024  152   4.3  4.6  (one cluster, TMEM)   1.84 1.89
//  128 1536  270   239  317  (CUDA cores)          5.4  6.0   (one part of the rank vector: 4.6 6.7)
//   48 1536  270             (CUDA cores)          2.98 3.12  (2.51 2.69)
//    9 1000  130             (CUDA cores)          2.38 2.44  (2.13 2.19)
LowRankRegPlan pick_lowrank_reg_plan(int B, int d, int r) {
  LowRankRegPlan best{};
  best.ok = false;
  const int kb1 = ((d + 31) / 32 + RR_WARPS - 1) / RR_WARPS;
  const int rt = (r + 15) / 16;
  const int kb2 = ((rt * 16 + 31) / 32 + RR_WARPS - 1) / RR_WARPS;
  // (a warp's range of two blocks must fit in a row)
  if (B < 1 || d < 64 || (d & 7) != 0 || kb1 > RR_MAX_KB || r < 1 || kb2 > 2) return best;
  const int sms = rec_reg_sms();
  const int mts[4] = {1, 2, 4, 6};
  for (int nt = 1; nt <= RR_MAX_NT; ++nt)
    for (int mt : mts) {
      const int ng = 8 * nt, groups = (B + ng - 1) / ng;
      int cpg = (d + 16 * mt - 1) / (16 * mt);
      if (cpg < rt) cpg = rt;
      if (cpg > sms || groups > REC_MAX_DB_ROWS) continue;
      const int fit = sms / cpg;
      const int launches = (groups + fit - 1) / fit;
      const int per = (groups + launches - 1) / launches;
      const int live = B < ng ? B : ng;
      const double kb_h = d * 2.0 * live / 1024, kb_q = rt * 32.0 * live / 1024;
      const double mb = per * live * 2e-6 * ((double)rt * d + (double)cpg * rt * 16);
      const double cost = launches * (2 * 680 + 11 * (kb_h + kb_q) + 18.0 * nt * (kb1 + mt * kb2) +
                                      36.0 * mt * nt + 43 * mb);
      if (!best.ok || cost < best.cost) {
        best.kb1 = (kb1 + 1) / 2 * 2; best.kb2 = kb2; best.mt = mt; best.nt = nt;
        best.cpg = cpg; best.rows = per * ng; best.cost = cost; best.ok = true;
      }
    }
  return best;
}

}  // namespace

bool lowrank_reg_supported(int T, int B, int d, int r) {
  return T >= 1 && options().rec_reg != 1 && options().rec_trace == 0 && pick_lowrank_reg_plan(B, d, r).ok;
}

int lowrank_reg(const LowRankRegArgs& a, cudaStream_t stream) {
  const LowRankRegPlan pl = pick_lowrank_reg_plan(a.B, a.d, a.r);
  if (!pl.ok) return ELMAN_ERR_UNSUPPORTED;
  const bool bwd = a.bwd != 0;
  // the rank vector with the bits that the kernel which had this shape before kept
  const bool split = !lowrank_tc_supported(a.T, a.B, a.d, a.r, a.bwd);
  const uintptr_t wide = (uintptr_t)a.state | (uintptr_t)a.q | (uintptr_t)a.q_low;
  const uintptr_t narrow = (uintptr_t)a.in0 | (uintptr_t)a.in1 | (uintptr_t)a.in2 | (uintptr_t)a.in3 |
                           (uintptr_t)a.out0 | (uintptr_t)a.out1;
  if ((wide & 15) != 0 || (narrow & 3) != 0 || (a.rq & 7) != 0) return ELMAN_ERR_UNSUPPORTED;
  LowRankRegKernel kern = (split ? (bwd ? lowrank_split_bwd_kernel : lowrank_split_fwd_kernel)
                                 : (bwd ? lowrank_reg_bwd_kernel : lowrank_reg_fwd_kernel))(pl.kb1, pl.kb2, pl.mt, pl.nt);
  if (kern == nullptr) return ELMAN_ERR_UNSUPPORTED;
  const size_t smem = lowrank_reg_smem(bwd, pl.kb1, pl.kb2, pl.mt, pl.nt, split);
  if (smem > 48 * 1024)
    ELMAN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  LowRankRegParams p{};
  p.T = a.T; p.B = a.B; p.d = a.d; p.r = a.r; p.r16 = (a.r + 15) / 16 * 16; p.rq = a.rq;
  p.cpg = pl.cpg;
  p.A1 = (const bf16*)a.A1; p.a1_row = a.a1_row; p.a1_k = a.a1_k;
  p.A2 = (const bf16*)a.A2; p.a2_row = a.a2_row; p.a2_k = a.a2_k;
  p.in0 = (const bf16*)a.in0; p.in1 = (const bf16*)a.in1;
  p.in2 = (const bf16*)a.in2; p.in3 = (const bf16*)a.in3;
  p.state = (bf16*)a.state; p.out0 = (bf16*)a.out0; p.out1 = (bf16*)a.out1; p.db = a.db;
  p.q = (bf16*)a.q; p.q_low = (bf16*)a.q_low;
  p.abort_word = a.sync;
  p.status = device_status_ptr();
  p.spin_limit = options().spin_limit;
  p.stall_step = (int)options().test_stall_step;
  // Cycles from a barrier to the first look at the state and at the rank vector: both exchanges
  // take longer, and looks that come too early delay them.  B = 32, d = 1536, r = 270, us per step:
  // 2.67 with no wait, 2.33 with these, 2.68 with 900 and 1200.
  p.hold = 600;
  p.hold_q = 600;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(((a.B < pl.rows ? a.B : pl.rows) + 8 * pl.nt - 1) / (8 * pl.nt) * pl.cpg);
  cfg.blockDim = dim3(RR_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  // the runtime's guarantee that the CTAs, which wait for one another, are resident together
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (!fits_together((const void*)kern, cfg)) return ELMAN_ERR_UNSUPPORTED;
  const size_t slot = (size_t)a.B * a.d * sizeof(bf16), q_slot = (size_t)a.B * a.rq * sizeof(bf16);
  ELMAN_CUDA_CHECK(cudaMemsetAsync(a.sync, 0, 4, stream));
  ELMAN_CUDA_CHECK(cudaMemsetAsync((char*)a.state + (bwd ? 0 : slot), 0xFF, a.T * slot, stream));
  ELMAN_CUDA_CHECK(cudaMemsetAsync((char*)a.q + (bwd ? q_slot : 0), 0xFF, a.T * q_slot, stream));
  if (split) ELMAN_CUDA_CHECK(cudaMemsetAsync(a.q_low, 0xFF, a.T * q_slot, stream));
  for (int b = 0; b < a.B; b += pl.rows) {
    p.b_lo = b;
    p.b_hi = b + pl.rows < a.B ? b + pl.rows : a.B;
    const int groups = (p.b_hi - b + 8 * pl.nt - 1) / (8 * pl.nt);
    cfg.gridDim = dim3(groups * pl.cpg);
    ELMAN_RETURN_IF(launch_together(kern, cfg, p));
    count_launch(true, REC_KERNEL_LOWRANK_REG);
  }
  const int rows = (a.B + 8 * pl.nt - 1) / (8 * pl.nt);
  if (bwd && rows > 1) return fold_db_rows(a.db, a.d, rows, stream);
  return ELMAN_OK;
}

}  // namespace elman
