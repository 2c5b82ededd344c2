// Low-rank recurrence with both factors in REGISTERS, bf16, warp-level tensor-core products.
//
//   forward   h_t  = tanh(U (V h_{t-1}) + pre_t),  y_t = h_t * silu(g_t)
//   backward  dv_t = (dy_t * silu(g_t) + V^T (U^T dv_{t+1})) * (1 - tanh(v_t)^2)
// (elman/cuda/lib/pure_lowrank_elman_fused_gpu.cu.cc:244-270, :355-501 of the reference)
//
// The machinery of rec_reg.cuh — batch groups of 8 NT rows, K split over eight warps, the tensor
// itself as the message — with two hand-offs per step.  The first ceil(r / 16) CTAs of a group own
// 16 rank rows each of the first factor: they read the group's state and publish their part of the
// rank vector, rounded to bf16, in `q`.  Every CTA owns 16 MT rows of the second factor, reads the
// rank vector (4.5 KB for 8 rows of rank 270) and finishes its features.  Both factors are read in
// place through row and column strides, so the backward pass needs no transposed copies; its rank
// vectors are U^T dv of every step but the first, which the weight gradients need as well and
// would otherwise compute again as a product over all T B rows.
//
// SPLIT: the rank vector in two bf16 parts, its rounded value and what the rounding left (16 bits of
// mantissa together).  The cluster kernel (lowrank_tc.cu) rounds the vector to bf16 between the two
// products, the CUDA-core kernel kept it in fp32; shapes that come from the latter (batches over 32,
// widths that are no multiple of 128, ranks too large for one cluster) take this form.  Relative error of
// h against 64 bits at T = 160, B = 128, d = 1536, r = 270: CUDA cores 2.748e-3, one part 2.930e-3, two
// parts 2.747e-3.  The second part costs 0.3 to 0.5 us of a step.  It is stored first, so whoever has seen
// the rounded value seldom waits for it.
//
// Bound, like the dense kernel's, by the chain: two L2 round trips per step.  Measured at B = 32,
// d = 1536, r = 270: see lowrank_reg.cu.
#pragma once

#include <float.h>

#include "rec_reg.cuh"

namespace elman {

struct LowRankRegParams : RecRegParams {
  int r, r16;                   // rank, and rank rounded up to the 16-row tiles
  int rq;                       // row stride of q
  const bf16* A1; long a1_row, a1_k;   // first factor [r, d]:  element (row, k) at row*a1_row + k*a1_k
  const bf16* A2; long a2_row, a2_k;   // second factor [d, r]
  bf16* q;                      // rank vectors [slots][B][rq]; slot of a step = slot of its input state
  bf16* q_low;                  // SPLIT: what rounding the entries of q to bf16 left, [T][B][rq]; slot = step
  int hold_q;                   // cycles from a CTA's last barrier to its first look at q
};

constexpr int LRR_PS1 = 20;     // row stride of the 16-row partial sums

// The first factor's fragments in shared memory instead of registers (8 KB1 of them): where both factors,
// both parts of the rank vector and the accumulators would spill.
__host__ __device__ constexpr bool lowrank_first_shared(int kb1, int kb2, int mt, bool split) {
  return split && (mt * kb2 > 8 || (kb1 == 8 && mt * kb2 >= 6));
}

inline size_t lowrank_reg_smem(bool bwd, int kb1, int kb2, int mt, int nt, bool split) {
  return rec_reg_smem(bwd, mt, nt) + (size_t)RR_WARPS * 8 * nt * LRR_PS1 * sizeof(float) +
         (lowrank_first_shared(kb1, kb2, mt, split) ? (size_t)kb1 * 2 * RR_THREADS * sizeof(uint4) : 0);
}

namespace rr {

// A fragments of rows row0 + {gq, gq + 8} over this warp's blocks of K, element by element.
template <int KB>
__device__ __forceinline__ void load_factor(uint32_t (&w)[KB][8], const bf16* A, long s_row, long s_k,
                                            int row0, int rows, const KRange<KB>& k, int K) {
  const unsigned short* a = reinterpret_cast<const unsigned short*>(A);
#pragma unroll
  for (int kb = 0; kb < KB; ++kb)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int row = row0 + 8 * u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t lo = 0, hi = 0;
        const int col = k.col + kb * 32 + 2 * j;
        if (row < rows && k.owns(kb)) {
          if (col < K) lo = __ldg(a + row * s_row + col * s_k);
          if (col + 1 < K) hi = __ldg(a + row * s_row + (col + 1) * s_k);
        }
        w[kb][2 * j + u] = lo | (hi << 16);
      }
    }
}

// What rounding a pair to bf16 left of it, as bf16; nothing of an entry that is no finite number.
__device__ __forceinline__ uint32_t rest(float2 v, uint32_t hi) {
  const float2 h = unpack(hi);
  return pack(fabsf(h.x) <= FLT_MAX ? v.x - h.x : 0.f, fabsf(h.y) <= FLT_MAX ? v.y - h.y : 0.f);
}

}  // namespace rr

template <bool BWD, int KB1, int KB2, int MT, int NT, bool SPLIT>
__global__ void __launch_bounds__(RR_THREADS, 1) lowrank_reg_kernel(const LowRankRegParams p) {
  constexpr int R = 16 * MT, NG = 8 * NT;
  constexpr int CH1 = NT == 1 ? 2 : 1, CH2 = MT * NT == 1 ? 2 : 1;
  constexpr bool W1S = lowrank_first_shared(KB1, KB2, MT, SPLIT);
  typedef rr::Tail<BWD, R, NG> Tail;
  constexpr int PS = Tail::PS;
  extern __shared__ __align__(16) float part[];   // [2][warps][NG][PS], ring, [warps][NG][LRR_PS1]
  __shared__ int s_bad[2][2];                     // [product][step parity]: a wait gave up

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int T = p.T, d = p.d;
  const int grp = blockIdx.x / p.cpg, c = blockIdx.x - grp * p.cpg;
  const int f0 = c * R, b0 = p.b_lo + grp * NG;
  const bool ranked = c * 16 < p.r;               // this CTA owns rank rows 16 c .. 16 c + 15
  if (tid < 4) s_bad[tid >> 1][tid & 1] = 0;

  const rr::KRange<KB1> k1(d, warp, tq);
  const rr::KRange<KB2> k2(p.r16, warp, tq);
  uint32_t w1[1][KB1][8], w2[MT][KB2][8];
  rr::load_factor<KB1>(w1[0], p.A1, p.a1_row, p.a1_k, c * 16 + gq, p.r, k1, d);
  // (every thread reads back its own)
  uint4* const w1_s = reinterpret_cast<uint4*>(part + 2 * RR_WARPS * NG * PS +
                                               RR_AHEAD * Tail::ITEMS * Tail::NIN * RR_THREADS +
                                               RR_WARPS * NG * LRR_PS1) + tid;
  if (W1S) {
#pragma unroll
    for (int kb = 0; kb < KB1; ++kb)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        w1_s[(kb * 2 + j) * RR_THREADS] = make_uint4(w1[0][kb][4 * j], w1[0][kb][4 * j + 1], w1[0][kb][4 * j + 2],
                                                     w1[0][kb][4 * j + 3]);
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
    rr::load_factor<KB2>(w2[mt], p.A2, p.a2_row, p.a2_k, f0 + mt * 16 + gq, d, k2, p.r);
  // a warp whose part of K is behind the rank has nothing to add, once and for all
  const bool busy = !SPLIT || warp * (KB2 * 32) < p.r16;
  if (!busy)
    for (int i = lane; i < 2 * NG * PS; i += 32) part[(i / (NG * PS) * RR_WARPS + warp) * NG * PS + i % (NG * PS)] = 0.f;
  uint32_t h_off[NT], q_off[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int b = min(b0 + nt * 8 + gq, p.b_hi - 1);
    h_off[nt] = (uint32_t)(b * d + k1.col) * 2u;
    q_off[nt] = (uint32_t)(b * p.rq + k2.col) * 2u;
  }

  float* const ring = part + 2 * RR_WARPS * NG * PS;
  float* const part1 = ring + RR_AHEAD * Tail::ITEMS * Tail::NIN * RR_THREADS;
  Tail tail(p, ring, f0, b0);
  const int slot = tail.slot, q_slot = p.B * p.rq * 2;
  const long step_bytes = BWD ? -(long)slot : (long)slot;
  long at = BWD ? (long)(T - 1) * slot : 0;
#pragma unroll
  for (int s = 0; s < RR_AHEAD - 1; ++s) tail.fetch(s, at + s * step_bytes);
  // the feature pair of my rank rows that this thread finishes
  const int n1 = tid >> 3, pair1 = tid & 7;
  const bool mine1 = tid < 8 * NG && b0 + n1 < p.b_hi;
  const uint32_t q_mine = (uint32_t)((b0 + n1) * p.rq + c * 16 + 2 * pair1) * 2u;
  const int stall_step = blockIdx.x == 0 ? p.stall_step : -1;
  uint32_t met = rr::cycles();
  __syncthreads();
  auto give_up = [&](int product, int s) {
    if (atomicExch(p.abort_word, 1) == 0) report_timeout(p.status, KID_LOWRANK_TC, s);
    s_bad[product][s & 1] = 1;
  };

  for (int s = 0; s < T; ++s, at += step_bytes) {
    tail.fetch(s + RR_AHEAD - 1, at + (RR_AHEAD - 1) * step_bytes);
    tail.premath(s);
    const long from = BWD ? T - s : s;            // time slot of the input state
    char* const q = reinterpret_cast<char*>(p.q) + from * q_slot;
    char* const q_low = reinterpret_cast<char*>(p.q_low) + (long)s * q_slot;
    if (ranked) {
      // ---- my 16 entries of the rank vector ----
      const char* src = reinterpret_cast<const char*>(p.state) + from * slot;
      while (rr::cycles() - met < (uint32_t)p.hold) { }
      uint4 x[NT][KB1];
      rr::look(x, src, h_off);
      if (s > 0 && !rr::await(x, src, h_off, s == stall_step, p.spin_limit, p.abort_word)) give_up(0, s);
      __syncwarp();
      if (W1S) {
#pragma unroll
        for (int kb = 0; kb < KB1; ++kb)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint4 v = w1_s[(kb * 2 + j) * RR_THREADS];
            w1[0][kb][4 * j] = v.x; w1[0][kb][4 * j + 1] = v.y;
            w1[0][kb][4 * j + 2] = v.z; w1[0][kb][4 * j + 3] = v.w;
          }
      }
      float acc[CH1][1][NT][4];
      rr::products(acc, w1, x);
      rr::put_partials(part1 + warp * NG * LRR_PS1, LRR_PS1, gq, tq, acc);
      __syncthreads();
      met = rr::cycles();
      const int bad = s_bad[0][s & 1];
      if (mine1) {
        const float2 v = rr::gather_pair(part1 + n1 * LRR_PS1 + 2 * pair1, NG * LRR_PS1);
        const uint32_t hi = rr::pack(v.x, v.y);
        if (SPLIT) rr::st_relaxed_u32(q_low + q_mine, rr::rest(v, hi));
        rr::st_relaxed_u32(q + q_mine, hi);
      }
      if (bad) break;
    }
    // ---- my features from the whole rank vector ----
    float* buf = part + (s & 1) * (RR_WARPS * NG * PS);
    if (busy) {
      while (rr::cycles() - met < (uint32_t)p.hold_q) { }
      uint4 x[NT][KB2], xl[NT][KB2];
      rr::look(x, q, q_off);
      if (SPLIT && KB2 == 1) rr::look(xl, q_low, q_off);   // (more blocks: a look that comes too early costs more)
      if (!rr::await(x, q, q_off, false, p.spin_limit, p.abort_word)) give_up(1, s);
      __syncwarp();
      if (SPLIT && KB2 > 1) rr::look(xl, q_low, q_off);
      float acc[CH2][MT][NT][4];
      rr::products(acc, w2, x);
      if (SPLIT) {
        if (!rr::await(xl, q_low, q_off, false, p.spin_limit, p.abort_word)) give_up(1, s);
        __syncwarp();
        rr::add_products(acc, w2, xl);
      }
      rr::put_partials(buf + warp * NG * PS, PS, gq, tq, acc);
    }
    __syncthreads();
    met = rr::cycles();
    const int bad = s_bad[1][s & 1];
    tail.publish(buf, at);
    tail.store_rest(at);
    if (bad) break;
  }
  if (BWD) tail.fold_bias(part, f0, p.b_lo / NG + grp);
}

}  // namespace elman
