// Plans and launches of the register-resident recurrence (rec_reg.cuh).
#include <limits.h>

#include <atomic>

#include "rec_reg_table.cuh"

namespace elman {

namespace {

struct RecRegPlan {
  int mt, kb, nt;
  int groups, cpg;        // batch groups, or sets of `turns` groups, that have CTAs of their own
  int turns;              // 0: no turns, rec_reg_kernel
  bool ok;
};

// MB of state that one look of all CTAs together reads.
double rr_look_mb(int B, int d, int cpg) { return (double)B * d * 2 * cpg / 1e6; }

// Cycles from a step's barrier to the first look at the next state.  What a warp with outputs has
// to do until then takes about 700; a look that comes too early costs its own round trip and the
// L2 bandwidth that the other CTAs' looks and stores need (d = 1280, B = 32, 108 CTAs: 1.60 us per
// step without the wait, 1.38 with 800 cycles; B = 3, 80 CTAs: 1.25 and 0.98 with 600).
int rr_hold(int B, int d, int cpg) {
  const double mb = rr_look_mb(B, d, cpg);
  const int cycles = mb < 0.5 ? 450 : (int)(560 + 110 * mb);
  return cycles > 1000 ? 1000 : cycles;
}

// Groups of 8 or 16 rows, 16 to 64 rows of W per CTA.  Time of a step in ns, fitted to all plans of
// ten shapes (B 3 to 64, d 256 to 2048; 5 % mean error): 680 for the hand-off through L2 and what
// follows the barrier, 11 per KB of state a CTA reads, 18 per m-tile, n-tile and K block (the
// tensor pipe does an m16n8k16 in 2 cycles per SM), 36 per m-tile and n-tile of partial sums, 43
// per MB that all CTAs read together.  Measured, us per step forward / backward:
//
//    B    d   TMEM kernel   NT MT CTAs   this kernel
//    3  1280   3.96 3.86     1  1   80   0.98 0.99
//   32  1280   4.27 4.39     1  4   80   1.47 1.54     (MT = 3, 108 CTAs: 1.38 1.43)
//   48   768   4.70 4.72     1  3   96   1.19 1.27
//   64  1280   5.37 5.49     2  3  108   2.04 2.12
//   32  2048   4.81 4.85     2  2  128   2.21 2.24
//   37   952    55   40      1  4   75   1.33 1.41     (no TMEM plan: CUDA cores)
//
// Among plans within 8 % of the best estimate the one with the fewest CTAs is taken: the SMs it
// leaves alone serve other streams.
RecRegPlan pick_rec_reg_plan(int B, int d) {
  RecRegPlan best{};
  best.ok = false;
  const int kb = ((d + 31) / 32 + RR_WARPS - 1) / RR_WARPS;
  if (B < 1 || B > RR_MAX_BATCH || d < 8 || (d & 7) != 0 || kb > RR_MAX_KB) return best;
  const int sms = rec_reg_sms();
  double best_cost = 0;
  for (int pass = 0; pass < 2; ++pass) {
    int best_ctas = 0;
    for (int nt = 1; nt <= RR_MAX_NT; ++nt)
      for (int mt = 1; mt <= RR_MAX_MT; ++mt) {
        if (mt * kb > RR_MAX_W) continue;
        const int groups = (B + 8 * nt - 1) / (8 * nt), cpg = (d + 16 * mt - 1) / (16 * mt);
        const int ctas = groups * cpg;
        if (ctas > sms || groups > REC_MAX_DB_ROWS) continue;
        const double in_kb = d * 2.0 * (B < 8 * nt ? B : 8 * nt) / 1024;
        const double cost = 680 + 11 * in_kb + 18.0 * mt * nt * kb + 36.0 * mt * nt +
                            43 * rr_look_mb(B, d, cpg);
        if (pass == 0) {
          if (best_cost == 0 || cost < best_cost) best_cost = cost;
        } else if (cost <= 1.08 * best_cost && (best_ctas == 0 || ctas < best_ctas)) {
          best_ctas = ctas;
          best.mt = mt; best.kb = kb; best.nt = nt; best.groups = groups; best.cpg = cpg;
          best.ok = true;
        }
      }
  }
  return best;
}

// Sets of batch groups, each on CTAs of its own and taking turns there, on at most `ctas` CTAs.
// (Copies of the grid over shares of the batch: option rec_replicas limits them as it does those of
// the TMEM kernel.)
RecRegPlan turns_plan(int T, int B, int d, int ctas) {
  RecRegPlan pl{};
  pl.kb = ((d + 31) / 32 + RR_WARPS - 1) / RR_WARPS;
  pl.ok = false;
  if (B < 1 || d < 8 || (d & 7) != 0 || pl.kb > RR_MAX_KB) return pl;
  pl.mt = rr::turns_mt(pl.kb);
  pl.nt = 1;
  pl.cpg = (d + 16 * pl.mt - 1) / (16 * pl.mt);
  const int groups = (B + 7) / 8;
  int sets = ctas / pl.cpg;
  if (sets > REC_MAX_DB_ROWS) sets = REC_MAX_DB_ROWS;
  if (options().rec_replicas > 0 && sets > options().rec_replicas) sets = (int)options().rec_replicas;
  sets = sets < 1 ? 1 : sets > groups ? groups : sets;
  pl.turns = (groups + sets - 1) / sets;
  pl.groups = (groups + pl.turns - 1) / pl.turns;
  if (pl.turns == 1) pl.turns = 0;
  // the kernel holds the bytes of a time slot and the number of turns in 32 bits
  pl.ok = pl.groups * pl.cpg <= rec_reg_sms() && (long)B * d < (1L << 30) &&
          (long)T * pl.turns <= INT_MAX - RR_AHEAD;
  return pl;
}

// The plan for callers that overlap launches: the most rows of W per CTA, and as many of the batch
// groups on one set of CTAs as make the launch a sixth of the device, so that six fit (the pipelined
// model runs up to one per layer).  Measured, one optimizer step in ms with one set / with two:
// d 1280 B 32, six layers, 20 / 40 CTAs 11.52 / 11.62; d 768 B 13, six layers, 12 / 24 CTAs 3.32 /
// 3.23; d 256 B 32, four layers, 4 / 8 CTAs 1.64 / 1.54.  Where every group has its own CTAs this
// is rec_reg_kernel; a plan with more CTAs than the fast one is of no use.
RecRegPlan pick_compact_plan(int T, int B, int d, const RecRegPlan& fast) {
  const RecRegPlan pl = turns_plan(T, B, d, rec_reg_sms() / 6);
  return pl.ok && pl.groups * pl.cpg <= fast.groups * fast.cpg ? pl : fast;
}

// Batches with more groups than the device has room for take turns on all of it, up to where the TMEM
// kernel, which needs about the same time for 64 rows as for 32, is ahead: 512 rows, or six turns where a
// CTA holds 32 rows of W instead of 64 or 48 (d > 1536).  us per step forward / backward, TMEM kernel and
// turns:
//
//    B    d   TMEM kernel    turns              B    d   TMEM kernel    turns
//   128   512   4.66  4.97   1.19  1.59        256  1536   8.55  9.09   6.70  7.26
//   256   768   5.18  5.44   2.39  2.54        512  1536  16.8  17.7   13.1  14.1
//   128  1024   5.69  5.75   2.14  2.31         64  2048   6.18  6.37   3.75  4.02
//   512  1024  14.9  15.4    6.59  6.92         96  2048   5.93  6.13   5.45  5.81
//   128  1280   5.66  5.91   2.96  3.17        128  2048   6.21  5.74   7.10  7.61
//   512  1280  10.7  10.1    9.15  9.60        256   952   350   235    3.51  3.77   (CUDA cores)
RecRegPlan plan_for(int T, int B, int d, int compact) {
  const RecRegPlan fast = pick_rec_reg_plan(B, d);
  if (fast.ok) return compact ? pick_compact_plan(T, B, d, fast) : fast;
  RecRegPlan pl = turns_plan(T, B, d, rec_reg_sms());
  const bool slow = compact || B > 512 || (pl.kb > 6 && pl.turns > 6);
  if (pl.ok && slow && rec_tc_supported(T, B, d, 0) && rec_tc_supported(T, B, d, 1)) pl.ok = false;
  return pl;
}

// Options that select a plan or a part of the TMEM kernel select that kernel (rec_replicas limits the
// copies of either grid).
bool rr_enabled() {
  const Options& o = options();
  return o.rec_reg != 1 && o.rec_ksplit == 0 && o.rec_groups == 0 && o.rec_mma_warps == 0 &&
         o.rec_trace == 0 && o.rec_w_tmem == 0 && o.rec_direct_publish == 0 && o.rec_large_batch == 1 &&
         o.rec_group_cap == 0 && o.rec_fin_groups == 0;
}

int rr_launch(bool bwd, const RecRegPlan& pl, RecRegParams& p, int* sync, int compact, cudaStream_t stream) {
  const bool turns = pl.turns > 0;
  RecRegKernel kern = turns ? (bwd ? rec_turns_bwd_kernel(pl.kb) : rec_turns_fwd_kernel(pl.kb))
                      : bwd ? rec_reg_bwd_kernel(pl.mt, pl.kb, pl.nt)
                            : rec_reg_fwd_kernel(pl.mt, pl.kb, pl.nt);
  // rows of W and of the state are read 16 bytes at a time, the rest in feature pairs (turns: fours)
  const uintptr_t wide = (uintptr_t)p.W | (uintptr_t)p.state;
  const uintptr_t narrow = (uintptr_t)p.in0 | (uintptr_t)p.in1 | (uintptr_t)p.in2 | (uintptr_t)p.in3 |
                           (uintptr_t)p.out0 | (uintptr_t)p.out1;
  if (kern == nullptr || (wide & 15) != 0 || (narrow & (turns ? 7 : 3)) != 0)
    return ELMAN_ERR_UNSUPPORTED;
  const size_t smem = turns ? rec_turns_smem(bwd, pl.mt) : rec_reg_smem(bwd, pl.mt, pl.nt);
  if (smem > 48 * 1024)
    ELMAN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // CTAs wait for one another.  A cooperative launch is the runtime's guarantee that they are
  // resident together, whatever else runs.  Callers that overlap launches (ELMAN_FLAG_COMPACT) go
  // without it, since it would hold a launch back until all of it fits at once: they run side by side
  // only what fits side by side, by elman_b200_recurrence_blocks, which is 0 under 128 features.
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(pl.groups * pl.cpg);
  cfg.blockDim = dim3(turns ? RR_TURN_THREADS : RR_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = compact && p.d >= RR_MIN_CONCURRENT_D ? 0 : 1;
  if (!fits_together((const void*)kern, cfg)) return ELMAN_ERR_UNSUPPORTED;
  p.b_lo = 0; p.b_hi = p.B;
  p.cpg = pl.cpg;
  p.turns = pl.turns;
  p.hold = rr_hold(p.B, p.d, pl.cpg);
  p.abort_word = sync;
  p.status = device_status_ptr();
  p.spin_limit = options().spin_limit;
  p.stall_step = (int)options().test_stall_step;
  ELMAN_CUDA_CHECK(cudaMemsetAsync(sync, 0, 4, stream));
  // every slot the kernel writes starts out as "not there yet"
  const size_t slot = (size_t)p.B * p.d * sizeof(bf16);
  ELMAN_CUDA_CHECK(cudaMemsetAsync((char*)p.state + (bwd ? 0 : slot), 0xFF, (size_t)p.T * slot, stream));
  ELMAN_RETURN_IF(launch_together(kern, cfg, p));
  count_launch(true, turns ? REC_KERNEL_TURNS : REC_KERNEL_REG);
  return ELMAN_OK;
}

}  // namespace

int rec_reg_sms() {
  static std::atomic<int> sms[64];     // any host thread
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return 0; }
  n = sms[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    sms[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

bool rec_reg_supported(int T, int B, int d, int compact) {
  return T >= 1 && rr_enabled() && plan_for(T, B, d, compact).ok;
}

int rec_reg_blocks(int T, int B, int d, int compact) {
  const RecRegPlan pl = plan_for(T, B, d, compact);
  return pl.ok && d >= RR_MIN_CONCURRENT_D ? pl.groups * pl.cpg : 0;
}

int rec_fwd_reg(const RecFwdArgs& a, cudaStream_t stream) {
  const RecRegPlan pl = plan_for(a.T, a.B, a.d, a.compact);
  if (!pl.ok) return ELMAN_ERR_UNSUPPORTED;
  RecRegParams p{};
  p.T = a.T; p.B = a.B; p.d = a.d;
  p.W = (const bf16*)a.W;
  p.in0 = (const bf16*)a.pre; p.in1 = (const bf16*)a.g;
  p.self_gate = a.g == nullptr ? 1 : 0;
  p.state = (bf16*)a.h; p.out0 = (bf16*)a.v; p.out1 = (bf16*)a.y;
  return rr_launch(false, pl, p, a.sync, a.compact, stream);
}

int rec_bwd_reg(const RecBwdArgs& a, cudaStream_t stream) {
  const RecRegPlan pl = plan_for(a.T, a.B, a.d, a.compact);
  if (!pl.ok) return ELMAN_ERR_UNSUPPORTED;
  RecRegParams p{};
  p.T = a.T; p.B = a.B; p.d = a.d;
  p.W = (const bf16*)a.Wt;
  p.self_gate = a.g == nullptr ? 1 : 0;
  p.in0 = (const bf16*)(a.g != nullptr ? a.g : a.dy); p.in1 = (const bf16*)a.dy;
  p.in2 = (const bf16*)a.h; p.in3 = (const bf16*)a.v;
  p.state = (bf16*)a.dv; p.out0 = (bf16*)a.dg; p.db = a.db;
  ELMAN_RETURN_IF(rr_launch(true, pl, p, a.sync, a.compact, stream));
  if (pl.groups > 1) return fold_db_rows(a.db, a.d, pl.groups, stream);
  return ELMAN_OK;
}

}  // namespace elman
