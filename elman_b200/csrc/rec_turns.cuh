// Dense recurrence with W in registers, several batch groups on one set of CTAs (see rec_reg.cuh):
// the groups take turns on the W that the CTAs hold, and one group's state is on its way through L2
// while the others' products run.
//
// For callers that overlap several recurrences, or a recurrence and other kernels, SMs held times
// duration is what counts: one group alone keeps its CTAs waiting for most of a step.  What bounds
// a turn (one step of one group) is then the latency of the instructions a warp runs one behind the
// other: 2000 cycles when eight warps do everything (products 390, look and check 350, partial sums
// 140, gathering and storing them 400, the inputs of later turns 600; d = 1280).  So the work is
// split: eight warps look, multiply and hand over partial sums, four more do all that follows, four
// features per thread, a turn behind them; the two sides meet on named barriers.
//
// us per step forward / backward, B = 32 (TMEM kernel's compact plan before): d 1280 on 20 CTAs
// 3.7 / 3.9 (5.2 / 5.3); the training step of six such layers 13.24 -> 11.5 ms.
#pragma once

#include "rec_reg.cuh"

namespace elman {

// Eight warps with W and four for what follows the products.
constexpr int RR_TAIL_THREADS = 128;
constexpr int RR_TURN_THREADS = RR_THREADS + RR_TAIL_THREADS;
// Registers of the two roles (setmaxnreg).  A block is launched with 168 per thread (65536 over 384
// threads, in steps of 8): 256 x 216 + 128 x 72 = 384 x 168.
constexpr int RR_TURN_REGS = 168, RR_MAIN_REGS = 216, RR_TAIL_REGS = 72;
static_assert(RR_THREADS * RR_MAIN_REGS + RR_TAIL_THREADS * RR_TAIL_REGS == RR_TURN_THREADS * RR_TURN_REGS,
              "the roles' registers must be those of the launch");
// named barriers: partial sums complete / read (two buffers each), the tail's own
constexpr int RR_BAR_FULL = 1, RR_BAR_FREE = 3, RR_BAR_TAIL = 5;

// Shared memory: two buffers of partial sums, and the ring of inputs.
inline size_t rec_turns_smem(bool bwd, int mt) {
  return (size_t)2 * RR_WARPS * 8 * (16 * mt + 4) * sizeof(float) +
         (size_t)RR_AHEAD * (bwd ? 4 : 2) * RR_TAIL_THREADS * sizeof(uint2);
}

namespace rr {

__device__ __forceinline__ void named_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void copy_quad(uint2* dst, const char* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(ptx::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void st_relaxed_v2(void* p, uint32_t a, uint32_t b) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}

// What follows the products of a turn, for one of the RR_TAIL_THREADS threads: four neighbouring
// features of one row (8 bytes of every tensor), the same ones in every group.  The arithmetic is
// that of Tail.  `first`: byte offset of the group's first row, `rows`: its rows inside the batch.
template <bool BWD, int R>
struct QuadTail {
  static constexpr int NG = 8;
  static constexpr int PS = R + 4;       // row stride of the partial sums
  static constexpr int QUADS = R / 4;
  static constexpr int NIN = BWD ? 4 : 2;
  static_assert(QUADS * NG <= RR_TAIL_THREADS, "one quad per thread");
  const RecRegParams& p;
  const int t, slot;
  uint2* const ring;
  int row;                // row in the group; past every group for a thread without a quad
  int spart;
  uint32_t off;           // byte offset inside one [B, d] slot, first group
  float e0[4], e1[4], dbs[4];   // as in Tail
  uint32_t late[2], o0[2], o1[2];

  __device__ __forceinline__ QuadTail(const RecRegParams& p_, int t_, float* ring_area, int f0, int b0)
      : p(p_), t(t_), slot(p_.B * p_.d * 2), ring(reinterpret_cast<uint2*>(ring_area) + t_) {
    const int n = t / QUADS, f = 4 * (t - n * QUADS);
    row = t < QUADS * NG && f0 + f < p.d ? n : NG;
    spart = row < NG ? n * PS + f : 0;
    off = row < NG ? (uint32_t)((b0 + n) * p.d + f0 + f) * 2u : 0u;
#pragma unroll
    for (int u = 0; u < 4; ++u) dbs[u] = 0.f;
  }
  __device__ __forceinline__ bool mine(int rows) const { return row < min(rows, NG); }
  static __device__ __forceinline__ const char* at_of(const bf16* base, long at, uint32_t o) {
    return reinterpret_cast<const char*>(base) + at + o;
  }
  __device__ __forceinline__ uint2* slot_of(int i, int k) const {
    return ring + ((i & (RR_AHEAD - 1)) * NIN + k) * RR_TAIL_THREADS;
  }
  // Inputs of turn i; `rows` 0 behind the last turn.
  __device__ __forceinline__ void fetch(int i, int rows, long at, uint32_t first) {
    if (mine(rows)) {
      const uint32_t o = off + first;
      copy_quad(slot_of(i, 0), at_of(p.in0, at, o));
      if (BWD || !p.self_gate) copy_quad(slot_of(i, 1), at_of(p.in1, at, o));
      if (BWD) {
        copy_quad(slot_of(i, 2), at_of(p.in2, at + slot, o));
        copy_quad(slot_of(i, 3), at_of(p.in3, at, o));
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // (a row past the batch works on what the ring holds; its results are never stored or summed)
  __device__ __forceinline__ void premath(int i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(RR_AHEAD - 1) : "memory");
    uint2 raw[NIN];
#pragma unroll
    for (int k = 0; k < NIN; ++k) raw[k] = *slot_of(i, k);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float2 a = unpack(u ? raw[0].y : raw[0].x), b = unpack(u ? raw[1].y : raw[1].x);
      float* const f0 = e0 + 2 * u;
      float* const f1 = e1 + 2 * u;
      if (!BWD) {
        f0[0] = a.x; f0[1] = a.y;
        if (!p.self_gate) { f1[0] = b.x * sigmoid_fast(b.x); f1[1] = b.y * sigmoid_fast(b.y); }
      } else {
        const float2 h = unpack(u ? raw[NIN - 2].y : raw[NIN - 2].x);
        const float2 v = unpack(u ? raw[NIN - 1].y : raw[NIN - 1].x);
        const float2 g = p.self_gate ? h : a;
        const float sx = sigmoid_fast(g.x), sy = sigmoid_fast(g.y);
        const float gx = b.x * h.x * sx * (1.f + g.x * (1.f - sx));
        const float gy = b.y * h.y * sy * (1.f + g.y * (1.f - sy));
        late[u] = pack(gx, gy);
        f0[0] = b.x * g.x * sx; f0[1] = b.y * g.y * sy;
        if (p.self_gate) { f0[0] += gx; f0[1] += gy; }   // d(h silu(h))/dh = silu(h) + h silu'(h)
        f1[0] = dtanh_from_v(v.x); f1[1] = dtanh_from_v(v.y);
      }
    }
    // computed now, not sunk to their use behind the barrier
#pragma unroll
    for (int u = 0; u < 4; ++u) asm volatile("" : "+f"(e0[u]), "+f"(e1[u]));
  }
  // The new state, from the partial sums in `buf`.
  __device__ __forceinline__ void publish(const float* buf, long at, uint32_t first, int rows) {
    if (!mine(rows)) return;
    float4 q[RR_WARPS];
#pragma unroll
    for (int wv = 0; wv < RR_WARPS; ++wv)
      q[wv] = *reinterpret_cast<const float4*>(buf + wv * (NG * PS) + spart);
#pragma unroll
    for (int st = 1; st < RR_WARPS; st *= 2)      // the order of gather_pair
#pragma unroll
      for (int wv = 0; wv < RR_WARPS; wv += 2 * st) {
        q[wv].x += q[wv + st].x; q[wv].y += q[wv + st].y;
        q[wv].z += q[wv + st].z; q[wv].w += q[wv + st].w;
      }
    const float a[4] = {q[0].x, q[0].y, q[0].z, q[0].w};
    char* dst = const_cast<char*>(at_of(p.state, BWD ? at : at + slot, off + first));
    float r[4];
    if (!BWD) {
#pragma unroll
      for (int u = 0; u < 4; ++u) r[u] = tanh_fast(a[u] + e0[u]);
      const uint32_t h01 = pack(r[0], r[1]), h23 = pack(r[2], r[3]);
      st_relaxed_v2(dst, h01, h23);
      o0[0] = pack(a[0] + e0[0], a[1] + e0[1]);
      o0[1] = pack(a[2] + e0[2], a[3] + e0[3]);
      if (p.self_gate) {     // the gate is the state as stored
        const float2 s01 = unpack(h01), s23 = unpack(h23);
        o1[0] = pack(r[0] * s01.x * sigmoid_fast(s01.x), r[1] * s01.y * sigmoid_fast(s01.y));
        o1[1] = pack(r[2] * s23.x * sigmoid_fast(s23.x), r[3] * s23.y * sigmoid_fast(s23.y));
      } else {
        o1[0] = pack(r[0] * e1[0], r[1] * e1[1]);
        o1[1] = pack(r[2] * e1[2], r[3] * e1[3]);
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) r[u] = (e0[u] + a[u]) * e1[u];
      st_relaxed_v2(dst, pack(r[0], r[1]), pack(r[2], r[3]));
#pragma unroll
      for (int u = 0; u < 4; ++u) dbs[u] += r[u];
      o0[0] = late[0]; o0[1] = late[1];
    }
  }
  // Outputs that no other CTA waits for.
  __device__ __forceinline__ void store_rest(long at, uint32_t first, int rows) {
    if (!mine(rows)) return;
    const uint32_t o = off + first;
    if (p.out0 != nullptr)
      *reinterpret_cast<uint2*>(const_cast<char*>(at_of(p.out0, at, o))) = make_uint2(o0[0], o0[1]);
    if (!BWD) *reinterpret_cast<uint2*>(const_cast<char*>(at_of(p.out1, at, o))) = make_uint2(o1[0], o1[1]);
  }
  // Bias gradient over the rows of all groups, in a fixed order (reuses the partial sums).
  __device__ __forceinline__ void fold_bias(float* part, int f0, int set) {
    named_sync(RR_BAR_TAIL, RR_TAIL_THREADS);
    if (row < NG) *reinterpret_cast<float4*>(part + spart) = make_float4(dbs[0], dbs[1], dbs[2], dbs[3]);
    named_sync(RR_BAR_TAIL, RR_TAIL_THREADS);
    if (t < R && f0 + t < p.d) {
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < NG; ++n) sum += part[n * PS + t];
      p.db[(long)set * p.d + f0 + t] = sum;
    }
  }
};

}  // namespace rr

template <bool BWD, int MT, int KB>
__global__ void __launch_bounds__(RR_TURN_THREADS, 1) rec_turns_kernel(const RecRegParams p) {
  constexpr int NT = 1, R = 16 * MT, NG = 8 * NT;
  constexpr int CH = MT * NT == 1 ? 2 : 1;
  typedef rr::QuadTail<BWD, R> Tail;
  constexpr int PS = Tail::PS;
  extern __shared__ __align__(16) float part[];   // [2][warps][NG][PS], then the ring of inputs
  // A wait of turn i gave up: noted in [i & 3], acted on by the tail behind its turn i + 1 and by
  // the others in front of the partial sums of turn i + 2 -- the same place for every warp, so no
  // barrier is left waiting.
  __shared__ volatile int s_bad[4];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int d = p.d;
  const int set = blockIdx.x / p.cpg, c = blockIdx.x - set * p.cpg;
  const int f0 = c * R, b0 = p.b_lo + set * p.turns * NG;
  const int groups = min(p.turns, (p.b_hi - b0 + NG - 1) / NG);
  const int total = p.T * groups, row_bytes = d * 2;
  const int slot = p.B * row_bytes;
  const long step_bytes = BWD ? -(long)slot : (long)slot;
  if (tid < 4) s_bad[tid] = 0;
  __syncthreads();

  // a place in the sequence of turns: all groups of a step, then the next step
  struct Place {
    int g;
    long at;
  };
  auto next = [&](Place& q) {
    if (++q.g == groups) { q.g = 0; q.at += step_bytes; }
  };
  Place now{0, BWD ? (long)(p.T - 1) * slot : 0};

  if (warp < RR_WARPS) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(RR_MAIN_REGS));
    const int gq = lane >> 2, tq = lane & 3;
    const rr::KRange<KB> k(d, warp, tq);
    uint32_t w[MT][KB][8];
    rr::load_weights(w, p.W, f0 + gq, d, k);
    const char* const base = reinterpret_cast<const char*>(p.state) + (BWD ? slot : 0) + k.col * 2;
    const int stall_turn = blockIdx.x == 0 && p.stall_step > 0 ? p.stall_step * groups : -1;
    const uint32_t none[NT] = {0};
    auto source = [&](const Place& q) {
      // a row past the batch reads the last row's state: its products are discarded
      return base + q.at + (long)(min(b0 + q.g * NG + gq, p.b_hi - 1) * row_bytes);
    };
    uint4 x[NT][KB];
    const char* src = source(now);
    rr::look(x, src, none);
    for (int i = 0; i < total; ++i) {
      // (the first slot was written before the launch, whatever it holds)
      if (i >= groups && !rr::await(x, src, none, i == stall_turn, p.spin_limit, p.abort_word)) {
        if (atomicExch(p.abort_word, 1) == 0)
          report_timeout(p.status, BWD ? KID_REC_TC_BWD : KID_REC_TC_FWD, i / groups);
        s_bad[i & 3] = 1;
      }
      __syncwarp();
      float acc[CH][MT][NT][4];
      rr::products(acc, w, x);
      if (i + 1 < total) {
        next(now);
        src = source(now);
        rr::look(x, src, none);
      }
      if (i >= 2) {
        rr::named_sync(RR_BAR_FREE + (i & 1), RR_TURN_THREADS);
        if (s_bad[(i - 2) & 3]) break;
      }
      rr::put_partials(part + (i & 1) * (RR_WARPS * NG * PS) + warp * NG * PS, PS, gq, tq, acc);
      rr::named_arrive(RR_BAR_FULL + (i & 1), RR_TURN_THREADS);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RR_TAIL_REGS));
    Tail tail(p, tid - RR_THREADS, part + 2 * RR_WARPS * NG * PS, f0, b0);
    auto first = [&](const Place& q) { return (uint32_t)(q.g * NG * row_bytes); };
    auto rows = [&](const Place& q) { return p.b_hi - b0 - q.g * NG; };
    Place fetched = now;
    for (int i = 0; i < RR_AHEAD - 1; ++i) {
      tail.fetch(i, i < total ? rows(fetched) : 0, fetched.at, first(fetched));
      next(fetched);
    }
    int bad = 0;
    for (int i = 0; i < total; ++i) {
      tail.fetch(i + RR_AHEAD - 1, i + RR_AHEAD - 1 < total ? rows(fetched) : 0, fetched.at, first(fetched));
      next(fetched);
      tail.premath(i);
      rr::named_sync(RR_BAR_FULL + (i & 1), RR_TURN_THREADS);
      const int last = bad;
      bad = s_bad[i & 3];
      tail.publish(part + (i & 1) * (RR_WARPS * NG * PS), now.at, first(now), rows(now));
      if (i + 2 < total && !last) rr::named_arrive(RR_BAR_FREE + (i & 1), RR_TURN_THREADS);
      tail.store_rest(now.at, first(now), rows(now));
      if (last) break;
      next(now);
    }
    if (BWD) tail.fold_bias(part, f0, set);
  }
}

}  // namespace elman
