// Dense recurrence with the recurrent matrix in REGISTERS, bf16, warp-level tensor-core products.
//
//   forward   h_t  = tanh(W h_{t-1} + pre_t),  y_t = h_t * silu(g_t)
//   backward  dv_t = (dy_t * silu(g_t) + W^T dv_{t+1}) * (1 - tanh(v_t)^2),  dg_t = dy_t h_t silu'(g_t)
// (elman/cuda/lib/mamba_gated_elman_gpu.cu.cc:451-473 forward, :527-558 backward of the reference)
//
// What bounds a recurrence of a few dozen sequences is the chain from one step to the next, not
// arithmetic or memory: at B = 32, d = 1280 a step is 105 MFLOP and 0.4 MB.  The chain here has
// as few links as an exchange between SMs allows:
//
//   * Sequences are independent, so the batch is cut into groups of 8 NT rows (8 = the narrowest
//     tensor-core operand); a group's CTAs exchange states with each other only.  A small group
//     is what keeps the exchange short: every CTA reads the group's whole state every step, 20 KB
//     at d = 1280 and 8 rows.
//   * CTA c of a group owns 16 MT rows of W.  Its eight warps split K; each keeps its part of W as
//     mma.sync A fragments in registers for the whole launch (MT x KB x 8 registers), so a step
//     loads nothing but the state.
//   * The state tensor itself is the message.  Its slots are filled with a pattern that no
//     conversion to bf16 produces (0xFFFF: the converter's NaN is 0x7FFF) before the launch; a
//     warp reads its K range of the next state straight into B fragments, again and again until no
//     word shows the pattern.  There is no flag, no fence, no barrier between CTAs and no staging
//     through shared memory: one store and one load through L2 are the whole hand-off.  K is
//     permuted inside blocks of 32 (the same way in W and in the state) so that a lane's two
//     k-steps of fragment are 16 contiguous bytes of a row.
//   * The eight partial sums meet in shared memory; after one CTA barrier each thread finishes one
//     or two feature pairs and stores them.  Everything else (gate, v, y, the inputs of later
//     steps) is off the chain.
//
// Where a step goes (B = 32, d = 1280, 80 CTAs, 1.47 us): about 0.7 us from a CTA's store to the
// data in the last reader's registers, 0.25 products, 0.1 partial sums out and in, 0.15 tanh and
// store; rec_reg.cu has the measurements against the TMEM kernel (4.3 us).
//
// Waits are bounded: a poll that runs out raises the abort word, every CTA leaves through the
// voting barrier of its step, and the status word names kernel and step.
#pragma once

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace elman {

constexpr int RR_WARPS = 8;
constexpr int RR_THREADS = 32 * RR_WARPS;
constexpr int RR_MAX_KB = 8;    // 32-column blocks of K per warp: d <= 2048
constexpr int RR_MAX_MT = 4;
constexpr int RR_MAX_W = 20;    // MT * KB: 160 registers of W per thread
constexpr int RR_MAX_NT = 2;
constexpr int RR_AHEAD = 4;     // steps of inputs in flight or waiting in shared memory

// Shared memory: two buffers of partial sums, and the ring of inputs.
inline size_t rec_reg_smem(bool bwd, int mt, int nt) {
  const int items = (8 * mt * 8 * nt + RR_THREADS - 1) / RR_THREADS;
  return ((size_t)2 * RR_WARPS * (8 * nt) * (16 * mt + 4) +
          (size_t)RR_AHEAD * items * (bwd ? 4 : 2) * RR_THREADS) * sizeof(float);
}

struct RecRegParams {
  int T, B, d;
  int b_lo, b_hi;         // batch rows of this launch
  int cpg;                // CTAs per batch group (rec_turns.cuh: per set of `turns` groups)
  int turns;
  const bf16* W;          // [d, d], row = output feature (backward: the transposed matrix)
  const bf16* in0;        // forward pre            backward g
  const bf16* in1;        // forward g              backward dy
  const bf16* in2;        //                        backward h [T+1 slots]
  const bf16* in3;        //                        backward v
  bf16* state;            // forward h [T+1 slots]  backward dv [T+1 slots]
  bf16* out0;             // forward v (or null)    backward dg (or null)
  bf16* out1;             // forward y
  float* db;              // backward: [groups][d] sums of dv
  int* abort_word;
  int* status;
  long spin_limit;
  int self_gate;          // no gate input: the state gates itself
  int hold;               // cycles from a step's barrier to the first look at the next state
  int stall_step;         // test hook: block 0 never sees its input of this step (-1 off)
};

namespace rr {

__device__ __forceinline__ uint4 ld_relaxed_v4(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u32(void* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void copy_word(uint32_t* dst, const unsigned int* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(ptx::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ uint32_t cycles() {
  uint32_t c;
  asm volatile("mov.u32 %0, %%clock;" : "=r"(c));
  return c;
}
__device__ __forceinline__ uint32_t largest(const uint4& v) { return max(max(v.x, v.y), max(v.z, v.w)); }
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Elementwise functions in hardware precision, as in the TMEM kernels; widths and batches that came from the
// CUDA-core kernel had tanhf and an IEEE division there.  Measured against 64 bits at those shapes: of 487 000
// values of h none rounds to another bf16 number (|x| from 0.05 to 3 times a normal variate), of h silu(z) 6 in
// 10^4 do (before: 1 in 10^5), its relative error is the same in five digits, and over whole sequences (200 x
// 37 x 952 and others) no output or gradient is further off than summation order makes it.  With tanhf and
// the division instead, 200 x 37 x 952 forward and backward takes 772 us instead of 703.
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sigmoid_fast(float z) { return __fdividef(1.f, 1.f + __expf(-z)); }
// 1 - tanh(v)^2 without cancellation: 4u/(1+u)^2 with u = exp(-2|v|)
__device__ __forceinline__ float dtanh_from_v(float v) {
  const float u = __expf(-2.f * fabsf(v));
  const float r = __fdividef(1.f, 1.f + u);
  return 4.f * u * r * r;
}
__device__ __forceinline__ float2 unpack(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// One look at a lane's fragments of the state: KB blocks of 32 columns for each of NT row tiles.
template <int NT, int KB>
__device__ __forceinline__ void look(uint4 (&x)[NT][KB], const char* src, const uint32_t (&x_off)[NT]) {
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) x[nt][kb] = ld_relaxed_v4(src + x_off[nt] + kb * 64);
}

// Looks again at what was not there yet until all of it is; false when the wait gave up.
// `stalled` (test hook): never satisfied.
template <int NT, int KB>
__device__ __forceinline__ bool await(uint4 (&x)[NT][KB], const char* src, const uint32_t (&x_off)[NT],
                                      bool stalled, long spin_limit, const int* abort_word) {
  long spins = 0;
  unsigned long long t_begin = 0;
  while (true) {
    // one comparison for everything: the pattern is the largest unsigned value
    uint32_t top = stalled ? 0xFFFFFFFFu : 0u;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) top = max(top, largest(x[nt][kb]));
    if (top != 0xFFFFFFFFu) return true;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int kb = 0; kb < KB; ++kb)
        if (largest(x[nt][kb]) == 0xFFFFFFFFu) x[nt][kb] = ld_relaxed_v4(src + x_off[nt] + kb * 64);
    if (++spins > spin_limit) return false;
    if ((spins & 63) == 0) {
      const unsigned long long now = ptx::globaltimer_ns();
      if (t_begin == 0) t_begin = now;
      if (ld_relaxed_gpu(abort_word) == 1 || now - t_begin > ptx::kWaitDeadlineNs) return false;
    }
  }
}

// The products of one warp: acc[mt][nt] += W tile mt (A fragments) times the state's row tile nt
// over KB blocks of two k-steps.
template <int CH, int MT, int NT, int KB>
__device__ __forceinline__ void add_products(float (&acc)[CH][MT][NT][4], const uint32_t (&w)[MT][KB][8],
                                             const uint4 (&x)[NT][KB]) {
#pragma unroll
  for (int kb = 0; kb < KB; ++kb) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
        mma_bf16(acc[0][mt][nt], w[mt][kb][0], w[mt][kb][1], w[mt][kb][2], w[mt][kb][3], x[nt][kb].x,
                 x[nt][kb].y);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
        mma_bf16(acc[CH - 1][mt][nt], w[mt][kb][4], w[mt][kb][5], w[mt][kb][6], w[mt][kb][7],
                 x[nt][kb].z, x[nt][kb].w);
  }
}

template <int CH, int MT, int NT, int KB>
__device__ __forceinline__ void products(float (&acc)[CH][MT][NT][4], const uint32_t (&w)[MT][KB][8],
                                         const uint4 (&x)[NT][KB]) {
#pragma unroll
  for (int ch = 0; ch < CH; ++ch)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[ch][mt][nt][u] = 0.f;
  add_products(acc, w, x);
}

// A warp's accumulators to its part of the partial-sum buffer [NT * 8 rows][stride].
template <int CH, int MT, int NT>
__device__ __forceinline__ void put_partials(float* dst, int stride, int gq, int tq,
                                             const float (&acc)[CH][MT][NT][4]) {
  float* mine = dst + 2 * tq * stride + gq;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float v = acc[0][mt][nt][u];
        if (CH == 2) v += acc[1][mt][nt][u];
        mine[(nt * 8 + (u & 1)) * stride + mt * 16 + 8 * (u >> 1)] = v;
      }
}

// Sum over the warps' partial sums of a feature pair.
__device__ __forceinline__ float2 gather_pair(const float* at, int warp_stride) {
  float2 q[RR_WARPS];
#pragma unroll
  for (int wv = 0; wv < RR_WARPS; ++wv) q[wv] = *reinterpret_cast<const float2*>(at + wv * warp_stride);
#pragma unroll
  for (int st = 1; st < RR_WARPS; st *= 2)
#pragma unroll
    for (int wv = 0; wv < RR_WARPS; wv += 2 * st) { q[wv].x += q[wv + st].x; q[wv].y += q[wv + st].y; }
  return q[0];
}

// The part of a step behind the products, for one thread: the feature pairs it finishes, their
// inputs (a ring of asynchronous copies) and their outputs.
template <bool BWD, int R, int NG>
struct Tail {
  static constexpr int PS = R + 4;       // row stride of the partial sums: conflict-free stores
  static constexpr int PAIRS = R / 2;
  static constexpr int ITEMS = (PAIRS * NG + RR_THREADS - 1) / RR_THREADS;   // pairs per thread
  static constexpr int NIN = BWD ? 4 : 2;
  const RecRegParams& p;
  const int slot;         // bytes of one time slot
  uint32_t* const ring;
  uint32_t off[ITEMS];    // byte offset inside one [B, d] slot
  int spart[ITEMS];       // offset of the pair's partial sums
  bool mine[ITEMS];
  // what does not depend on the recurrent term: forward e0 = pre, e1 = silu(g);
  // backward e0 = dy silu(g), e1 = 1 - tanh(v)^2, late = dg
  float2 e0[ITEMS], e1[ITEMS], dbs[ITEMS];
  uint32_t late[ITEMS], o0[ITEMS], o1[ITEMS];

  __device__ __forceinline__ Tail(const RecRegParams& p_, float* ring_area, int f0, int b0)
      : p(p_), slot(p_.B * p_.d * 2), ring(reinterpret_cast<uint32_t*>(ring_area) + threadIdx.x) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int e = threadIdx.x + i * RR_THREADS;
      const int n = e / PAIRS, f = 2 * (e - n * PAIRS);
      mine[i] = e < PAIRS * NG && f0 + f < p.d && b0 + n < p.b_hi;
      spart[i] = mine[i] ? n * PS + f : 0;
      off[i] = mine[i] ? (uint32_t)((b0 + n) * p.d + f0 + f) * 2u : 0u;
      dbs[i] = make_float2(0.f, 0.f);
    }
  }
  static __device__ __forceinline__ const unsigned int* word(const bf16* base, long at, uint32_t off) {
    return reinterpret_cast<const unsigned int*>(reinterpret_cast<const char*>(base) + at + off);
  }
  __device__ __forceinline__ uint32_t* slot_of(int s, int i, int k) const {
    return ring + (((s & (RR_AHEAD - 1)) * ITEMS + i) * NIN + k) * RR_THREADS;
  }
  // Inputs of step s (time slot at byte `at`).  Each thread copies its own words, RR_AHEAD - 1
  // steps ahead: loads into registers would share the scoreboards that the looks at the state
  // wait on, and tie the chain to DRAM.
  __device__ __forceinline__ void fetch(int s, long at) {
    if (s < p.T) {
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (mine[i]) {
          copy_word(slot_of(s, i, 0), word(p.in0, at, off[i]));
          if (BWD || !p.self_gate) copy_word(slot_of(s, i, 1), word(p.in1, at, off[i]));
          if (BWD) {
            copy_word(slot_of(s, i, 2), word(p.in2, at + slot, off[i]));
            copy_word(slot_of(s, i, 3), word(p.in3, at, off[i]));
          }
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void premath(int s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(RR_AHEAD - 1) : "memory");
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (!mine[i]) continue;
      uint32_t raw[NIN];
#pragma unroll
      for (int k = 0; k < NIN; ++k) raw[k] = *slot_of(s, i, k);
      if (!BWD) {
        e0[i] = unpack(raw[0]);
        if (!p.self_gate) {
          const float2 g = unpack(raw[1]);
          e1[i] = make_float2(g.x * sigmoid_fast(g.x), g.y * sigmoid_fast(g.y));
        }
      } else {
        float2 g = unpack(raw[0]);
        const float2 dy = unpack(raw[1]), h = unpack(raw[NIN - 2]), v = unpack(raw[NIN - 1]);
        if (p.self_gate) g = h;
        const float sx = sigmoid_fast(g.x), sy = sigmoid_fast(g.y);
        const float gx = dy.x * h.x * sx * (1.f + g.x * (1.f - sx));
        const float gy = dy.y * h.y * sy * (1.f + g.y * (1.f - sy));
        late[i] = pack(gx, gy);
        e0[i] = make_float2(dy.x * g.x * sx, dy.y * g.y * sy);
        if (p.self_gate) { e0[i].x += gx; e0[i].y += gy; }   // d(h silu(h))/dh = silu(h) + h silu'(h)
        e1[i] = make_float2(dtanh_from_v(v.x), dtanh_from_v(v.y));
      }
      // computed now, not sunk to their use behind the wait
      asm volatile("" : "+f"(e0[i].x), "+f"(e0[i].y), "+f"(e1[i].x), "+f"(e1[i].y));
      if (BWD) asm volatile("" : "+r"(late[i]));
    }
  }
  // The new state of the step whose time slot is at byte `at`, from the partial sums in `buf`.
  __device__ __forceinline__ void publish(const float* buf, long at) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (!mine[i]) continue;
      float2 a = gather_pair(buf + spart[i], NG * PS);
      char* dst = reinterpret_cast<char*>(p.state) + (BWD ? at : at + slot) + off[i];
      if (!BWD) {
        a.x += e0[i].x; a.y += e0[i].y;
        const float h0 = tanh_fast(a.x), h1 = tanh_fast(a.y);
        const uint32_t hp = pack(h0, h1);
        st_relaxed_u32(dst, hp);
        o0[i] = pack(a.x, a.y);
        if (p.self_gate) {     // the gate is the state as stored
          const float2 hs = unpack(hp);
          o1[i] = pack(h0 * hs.x * sigmoid_fast(hs.x), h1 * hs.y * sigmoid_fast(hs.y));
        } else {
          o1[i] = pack(h0 * e1[i].x, h1 * e1[i].y);
        }
      } else {
        const float d0 = (e0[i].x + a.x) * e1[i].x, d1 = (e0[i].y + a.y) * e1[i].y;
        st_relaxed_u32(dst, pack(d0, d1));
        dbs[i].x += d0; dbs[i].y += d1;
        o0[i] = late[i];
      }
    }
  }
  // Outputs that no other CTA waits for.
  __device__ __forceinline__ void store_rest(long at) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (!mine[i]) continue;
      if (p.out0 != nullptr) *const_cast<unsigned int*>(word(p.out0, at, off[i])) = o0[i];
      if (!BWD) *const_cast<unsigned int*>(word(p.out1, at, off[i])) = o1[i];
    }
  }
  // Bias gradient of the group's rows, in a fixed order (all threads; reuses the partial sums).
  __device__ __forceinline__ void fold_bias(float* part, int f0, int grp) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int e = threadIdx.x + i * RR_THREADS, n = e / PAIRS;
      if (e < PAIRS * NG) *reinterpret_cast<float2*>(part + n * PS + 2 * (e - n * PAIRS)) = dbs[i];
    }
    __syncthreads();
    if (threadIdx.x < R && f0 + (int)threadIdx.x < p.d) {
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < NG; ++n) sum += part[n * PS + threadIdx.x];
      p.db[(long)grp * p.d + f0 + threadIdx.x] = sum;
    }
  }
};

// The columns a lane reads: the warps' ranges of KB blocks cover [0, K) from the left; one that
// would reach past K is moved back and its columns that another warp owns get zero weights, so
// every look is in range without a predicate (K >= 32 KB, or KB = 1).  Lane tq takes columns 8 tq .. 8 tq + 7 of a block
// as fragment elements (k-step 0: b0, b1; k-step 1: b0, b1), two columns each.
template <int KB>
struct KRange {
  int own;      // first column that is this warp's
  int col;      // this lane's column in the first block
  bool any;     // false only when K < 32 leaves this lane nothing
  __device__ __forceinline__ KRange(int K, int warp, int tq) {
    own = warp * (KB * 32);
    col = min(own, max(0, K - KB * 32)) + tq * 8;
    any = col < K;
    if (!any) col = 0;
  }
  __device__ __forceinline__ bool owns(int kb) const { return any && col + kb * 32 >= own; }
};

// A lane's A fragments of MT tiles of W [d, d] from row `row0` on, over the warp's K range.
template <int MT, int KB>
__device__ __forceinline__ void load_weights(uint32_t (&w)[MT][KB][8], const bf16* W, int row0, int d,
                                             const KRange<KB>& k) {
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int kb = 0; kb < KB; ++kb)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int row = row0 + mt * 16 + 8 * u;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (row < d && k.owns(kb))
          x = __ldg(reinterpret_cast<const uint4*>(W + (long)row * d + k.col + kb * 32));
        w[mt][kb][0 + u] = x.x; w[mt][kb][2 + u] = x.y;
        w[mt][kb][4 + u] = x.z; w[mt][kb][6 + u] = x.w;
      }
}

}  // namespace rr

template <bool BWD, int MT, int KB, int NT>
__global__ void __launch_bounds__(RR_THREADS, 1) rec_reg_kernel(const RecRegParams p) {
  constexpr int R = 16 * MT;             // rows of W (features) of this CTA
  constexpr int NG = 8 * NT;             // batch rows of the group
  constexpr int CH = MT * NT == 1 ? 2 : 1;   // accumulator chains when one tile alone would serialise
  typedef rr::Tail<BWD, R, NG> Tail;
  constexpr int PS = Tail::PS;
  extern __shared__ __align__(16) float part[];   // [2][warps][NG][PS], then the ring of inputs
  __shared__ int s_bad[2];                        // a wait of an even / odd step gave up

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int T = p.T, d = p.d;
  const int grp = blockIdx.x / p.cpg, c = blockIdx.x - grp * p.cpg;
  const int f0 = c * R, b0 = p.b_lo + grp * NG;
  if (tid < 2) s_bad[tid] = 0;

  // ---- my part of W, once: rows f0 .. f0+R, this warp's KB blocks of 32 columns ----
  const rr::KRange<KB> k(d, warp, tq);
  uint32_t w[MT][KB][8];
  rr::load_weights(w, p.W, f0 + gq, d, k);
  // a row past the batch reads the last row's state: its products are discarded
  uint32_t x_off[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
    x_off[nt] = (uint32_t)(min(b0 + nt * 8 + gq, p.b_hi - 1) * d + k.col) * 2u;

  Tail tail(p, part + 2 * RR_WARPS * NG * PS, f0, b0);
  // running byte position of the step's slot in [T]-shaped tensors
  const int slot = tail.slot;
  const long step_bytes = BWD ? -(long)slot : (long)slot;
  long at = BWD ? (long)(T - 1) * slot : 0;
#pragma unroll
  for (int s = 0; s < RR_AHEAD - 1; ++s) tail.fetch(s, at + s * step_bytes);
  const int stall_step = blockIdx.x == 0 ? p.stall_step : -1;
  uint32_t met = rr::cycles();      // when this CTA's partial sums last met
  __syncthreads();

  for (int s = 0; s < T; ++s, at += step_bytes) {
    // ---- the step-local part of this step's arithmetic, then my K range of the group's state:
    // straight into fragments, until all of it is there ----
    tail.fetch(s + RR_AHEAD - 1, at + (RR_AHEAD - 1) * step_bytes);
    tail.premath(s);
    const char* src = reinterpret_cast<const char*>(p.state) + (BWD ? at + slot : at);
    while (rr::cycles() - met < (uint32_t)p.hold) { }
    uint4 x[NT][KB];
    rr::look(x, src, x_off);
    // (the first slot was written before the launch, whatever it holds)
    if (s > 0 && !rr::await(x, src, x_off, s == stall_step, p.spin_limit, p.abort_word)) {
      if (atomicExch(p.abort_word, 1) == 0)
        report_timeout(p.status, BWD ? KID_REC_TC_BWD : KID_REC_TC_FWD, s);
      s_bad[s & 1] = 1;
    }
    __syncwarp();
    float acc[CH][MT][NT][4];
    rr::products(acc, w, x);
    // ---- partial sums of the eight K ranges meet in shared memory (two buffers: the barrier of
    // the next step separates this buffer's readers from its next writers) ----
    float* buf = part + (s & 1) * (RR_WARPS * NG * PS);
    rr::put_partials(buf + warp * NG * PS, PS, gq, tq, acc);
    __syncthreads();
    met = rr::cycles();
    const int bad = s_bad[s & 1];
    tail.publish(buf, at);
    tail.store_rest(at);
    if (bad) break;
  }
  if (BWD) tail.fold_bias(part, f0, p.b_lo / NG + grp);
}

}  // namespace elman
