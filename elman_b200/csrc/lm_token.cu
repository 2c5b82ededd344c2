// One token for every sequence through a whole stack of E1 layers — the generation step of the
// byte-level model — as two launches:
//
//   residual add + RMSNorm -> in_proj, split, silu -> W_x x + W_h h + b, tanh, gate -> out_proj
// per layer, then the final norm and the tied head (elman/models/ladder_lm.py:986-1062,
// elman/models/mamba_gated_elman.py:283-306 of the reference, one framework op or cuBLAS call each).
//
// A token reads every weight once (98 MB at d = 1280, 6 layers: 15 us of HBM time) and does next to
// nothing with it, so what a step costs is its chain of products: three per layer, each needing all
// of the previous one's output.  The chain runs inside one kernel:
//
//   * CTA c owns features 16c .. 16c+15 of every matrix of every layer; eight sequences are the
//     narrow side of mma.m16n8k16.  What a feature needs of itself later — fp32 residual, gate —
//     stays in the thread that finishes it.
//   * Activations go from CTA to CTA as in rec_reg.cuh: buffers filled with a pattern no
//     conversion produces, read until it is gone.  No grid barrier.
//   * Eight warps split K.  A CTA's rows of in_proj, W_x and out_proj come into shared memory by
//     bulk copies a whole layer ahead — a slot is refilled as soon as its product is done — so the
//     memory system streams at its own pace behind the chain.  (With the weights loaded behind
//     each exchange instead, every product waited for DRAM and address translation: 105 us.)
//     W_h h is taken while the layer below is still on its way, and the RMSNorm happens on the
//     fragments: it costs a barrier, but no pass and no exchange of its own.
//
// Spectral normalisation of W_h scales its fragments as they are loaded.  The power iteration of all
// layers runs before it in a launch of its own: each matrix is cut by rows over a share of the SMs,
// stays in shared memory for all six products, and the vectors go through L2 the same way.
//
// Measured, d = 1280, 6 layers, us of GPU time per token of 1 / 27 / 64 sequences: 45 / 104 / 205, with
// the power iterations 70 / 130 / 230 (layer by layer 1540 / 1580 as issued from Python, about 1000 on
// the GPU).  At 1 sequence a product costs 2 us of hand-off and barriers; at 27 and more it is bound
// by the 80 CTAs reading every activation row (5.5 MB per product at 27) and by mma.sync.

#include "rec_reg.cuh"

namespace elman {

namespace {

constexpr int LT_MAX_LAYERS = 32;
// The dynamic shared memory of the two kernels depends on the sizes, the limit they are launched under
// must not: it belongs to the kernel, and another thread may set it between this one's setting and
// launch.  So every call sets the same limit (the token kernel keeps 2 KB for its static arrays).
constexpr int LT_SMEM_LIMIT = 225 * 1024, SP_SMEM_LIMIT = 220 * 1024;
constexpr int LT_MAX_ROWS = 64;
constexpr int LT_THREADS = 256;

struct LayerRefs {
  const bf16* norm; const bf16* w_in; const bf16* w_x; const bf16* w_h; const bf16* bias;
  const bf16* w_out; const bf16* h_prev; bf16* h_out; const float* scale;
};

struct LmTokenParams {
  int L, B, d, V;
  const long long* tokens;
  const bf16* embedding;
  const bf16* norm; const bf16* head;
  float eps;
  bf16* rb;        // [L][B][d]  residual after layer l, rounded (the next layer's norm input)
  bf16* xa;        // [L][B][d]  silu(x half of in_proj)
  bf16* y;         // [L][B][d]  gated cell output
  bf16* logits;    // [B][V]
  int* abort_word;
  int* status;
  long spin_limit;
  int stall_layer; // test hook: block 0 never sees this layer's input (-1 off)
  LayerRefs layer[LT_MAX_LAYERS];
};

// A fragments of 16 rows of a [rows, d] matrix in global memory, KB blocks of K.
template <int KB>
__device__ __forceinline__ void load_rows(uint32_t (&w)[1][KB][8], const bf16* W, int row0, int rows, int d,
                                          int gq, const rr::KRange<KB>& k) {
#pragma unroll
  for (int kb = 0; kb < KB; ++kb)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint4 x = make_uint4(0, 0, 0, 0);
      if (row0 + gq + 8 * u < rows && k.owns(kb))
        x = __ldg(reinterpret_cast<const uint4*>(W + (long)(row0 + gq + 8 * u) * d + k.col + kb * 32));
      w[0][kb][u] = x.x; w[0][kb][2 + u] = x.y; w[0][kb][4 + u] = x.z; w[0][kb][6 + u] = x.w;
    }
}

// two elements of the RMSNorm: x * rs * w, rounded once
__device__ __forceinline__ uint32_t normed(uint32_t x, uint32_t w, float rs) {
  const float2 a = rr::unpack(x), b = rr::unpack(w);
  return rr::pack(a.x * rs * b.x, a.y * rs * b.y);
}
__device__ __forceinline__ uint32_t scaled(uint32_t w, float s) {
  const float2 a = rr::unpack(w);
  return rr::pack(a.x * s, a.y * s);
}
__device__ __forceinline__ float square_sum(const uint4& v) {
  const float2 a = rr::unpack(v.x), b = rr::unpack(v.y), c = rr::unpack(v.z), e = rr::unpack(v.w);
  return ((a.x * a.x + a.y * a.y) + (b.x * b.x + b.y * b.y)) + ((c.x * c.x + c.y * c.y) + (e.x * e.x + e.y * e.y));
}
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// The CTA's rows of four matrices in shared memory, each row on a stride that puts neighbouring rows
// half a bank cycle apart; two norm weights; the partial sums.
constexpr int LT_R = 16, LT_PS = LT_R + 4;
__host__ __device__ inline int lt_row_bytes(int d) { return 2 * d + (64 - (2 * d) % 128 + 128) % 128; }
inline size_t lt_smem(int d, int nt) {
  return (size_t)4 * LT_R * lt_row_bytes(d) + (size_t)2 * 2 * d +
         (size_t)2 * RR_WARPS * 8 * nt * LT_PS * sizeof(float);
}

// Waits for the copies that were last sent for, by group.  A call: inlined, the path that no launch should
// take costs the kernel 36 more bytes of spills and 2 % of its time at 27 sequences.
__device__ __noinline__ void land(uint64_t* landed, const int* sent) {
  int none = 0;
  if (threadIdx.x < 3) ptx::mbar_wait(&landed[threadIdx.x], (uint32_t)sent[threadIdx.x] & 1u, 1L << 40, &none);
}

template <int KB, int NT, int TURNS>
__global__ void __launch_bounds__(LT_THREADS, 1) lm_token_kernel(const __grid_constant__ LmTokenParams p) {
  constexpr int ROWS = 8 * NT;              // sequences of a turn
  __shared__ __align__(16) float ss[ROWS][RR_WARPS];          // the norm's partial square sums
  __shared__ __align__(8) uint64_t landed[3];                 // in_proj, W_x, out_proj rows of a layer
  __shared__ int s_bad[2];
  __shared__ int s_abort;
  __shared__ int s_sent[3];                                   // layer last sent for, by group
  extern __shared__ __align__(128) uint8_t lt_dyn[];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int B = p.B, d = p.d, L = p.L;
  const int f0 = blockIdx.x * LT_R, rows_here = min(LT_R, d - f0);
  const int row_bytes = lt_row_bytes(d);
  bf16* const s_norm = reinterpret_cast<bf16*>(lt_dyn + 4 * LT_R * row_bytes);   // [2][d], by layer parity
  float* const part = reinterpret_cast<float*>(s_norm + 2 * d);   // [x | z][warp][ROWS][LT_PS]
  const rr::KRange<KB> k(d, warp, tq);
  // the feature pair this thread finishes in every turn
  const int e_row = tid >> 3, e_f = 2 * (tid & 7);
  const bool e_on = tid < ROWS * 8 && e_f < rows_here;
  if (tid == 0) {
    s_bad[0] = s_bad[1] = s_abort = 0;
    for (int i = 0; i < 3; ++i) ptx::mbar_init(&landed[i], 1);
    ptx::mbar_fence_init();
  }
  // rows past the matrix stay zero
  for (int i = tid; i < 4 * (LT_R - rows_here) * (row_bytes / 16); i += LT_THREADS) {
    const int r = i / (row_bytes / 16), slot = r / (LT_R - rows_here), row = rows_here + r % (LT_R - rows_here);
    *reinterpret_cast<uint4*>(lt_dyn + (slot * LT_R + row) * row_bytes + (i % (row_bytes / 16)) * 16) = make_uint4(0, 0, 0, 0);
  }
  __syncthreads();

  // ---- weights: slots 0, 1 the x and z rows of in_proj, 2 W_x, 3 out_proj ----
  // Rows of layer l on their way into a group's slots (group 0: in_proj, 1: W_x, 2: out_proj), one
  // bulk copy per row, by the last warp; the caller knows that nobody reads the slots any more.
  auto send_for = [&](int group, int l) {
    if (l >= L || warp != RR_WARPS - 1) return;
    const LayerRefs& r = p.layer[l];
    const uint32_t bytes = (uint32_t)d * 2u;
    if (lane == 0) {
      s_sent[group] = l;
      ptx::mbar_arrive_expect_tx(&landed[group], (uint32_t)((group == 0 ? 2 : 1) * rows_here) * bytes);
    }
    __syncwarp();
    const int slot = group == 0 ? lane >> 4 : group + 1, row = lane & 15;
    if ((group == 0 || lane < 16) && row < rows_here) {
      const bf16* src = group == 0 ? r.w_in + (long)slot * d * d : group == 1 ? r.w_x : r.w_out;
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(ptx::smem_u32(lt_dyn + (slot * LT_R + row) * row_bytes)), "l"(src + (long)(f0 + row) * d),
                     "r"(bytes), "r"(ptx::smem_u32(&landed[group]))
                   : "memory");
    }
    __syncwarp();
  };
  auto slot_rows = [&](uint32_t (&w)[1][KB][8], int slot) {    // its A fragments
#pragma unroll
    for (int kb = 0; kb < KB; ++kb)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        uint4 x = *reinterpret_cast<const uint4*>(lt_dyn + (slot * LT_R + gq + 8 * u) * row_bytes + (k.col + kb * 32) * 2);
        if (!k.owns(kb)) x = make_uint4(0, 0, 0, 0);
        w[0][kb][u] = x.x; w[0][kb][2 + u] = x.y; w[0][kb][4 + u] = x.z; w[0][kb][6 + u] = x.w;
      }
  };

  int turn = 0;                              // exchanges so far: flag parity
  bool dead = false;
  auto give_up = [&](int l) {
    if (atomicExch(p.abort_word, 1) != 1) report_timeout(p.status, KID_LM_TOKEN, l);
    s_bad[turn & 1] = 1;
  };
  auto await_rows = [&](int group, int l) {
    if (!ptx::mbar_wait(&landed[group], (uint32_t)l & 1u, p.spin_limit, &s_abort)) give_up(l);
  };
  uint32_t x_off[TURNS][NT];                 // a row past the batch reads the last one
#pragma unroll
  for (int t = 0; t < TURNS; ++t)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      x_off[t][nt] = (uint32_t)(min(t * ROWS + nt * 8 + gq, B - 1) * d + k.col) * 2u;
  // partial sums out (half 1: the z rows of in_proj)
  auto put = [&](int half, const float (&acc)[1][1][NT][4]) {
    rr::put_partials(part + (half * RR_WARPS + warp) * ROWS * LT_PS, LT_PS, gq, tq, acc);
  };
  auto pair_total = [&](int half) {
    return rr::gather_pair(part + half * RR_WARPS * ROWS * LT_PS + e_row * LT_PS + e_f, ROWS * LT_PS);
  };
  auto store_pair = [&](bf16* buf, int row, float x, float y) {
    rr::st_relaxed_u32(buf + (long)row * d + f0 + e_f, rr::pack(x, y));
  };
  // by the warps that finish fewest pairs, without waiting (settled before a later barrier)
  auto stage_norm = [&](int l) {
    const bf16* w = l < L ? p.layer[l].norm : p.norm;
    if (tid >= LT_THREADS / 2)
      for (int i = (tid - LT_THREADS / 2) * 8; i < d; i += LT_THREADS / 2 * 8)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                     ::"r"(ptx::smem_u32(s_norm + (l & 1) * d + i)), "l"(w + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto settle_norm = [&]() { asm volatile("cp.async.wait_group 0;" ::: "memory"); };
  // A token outside the vocabulary is reported through the status word and read as the nearest one.
  auto token = [&](int row) {
    const long long tok = p.tokens[row];
    return tok < 0 ? 0LL : tok >= p.V ? (long long)p.V - 1 : tok;
  };

  send_for(0, 0); send_for(1, 0); send_for(2, 0);
  stage_norm(0);
  // what the layers need besides: into L2, by one CTA each
  if ((int)blockIdx.x < L && tid == 0) {
    const LayerRefs& r = p.layer[blockIdx.x];
    prefetch_l2(r.norm, (uint32_t)d * 2u);
    if (r.h_prev != nullptr) prefetch_l2(r.h_prev, (uint32_t)(B * d) * 2u);
  }
  auto prefetch_w_h = [&](int l) {
    if (l < L && tid == LT_THREADS - 1 && p.layer[l].h_prev != nullptr)
      prefetch_l2(p.layer[l].w_h + (long)f0 * d, (uint32_t)(rows_here * d) * 2u);
  };
  prefetch_w_h(1);
  if (blockIdx.x == 0 && tid < B && token(tid) != p.tokens[tid])
    report_timeout(p.status, KID_LM_TOKEN, 0xFFFFFE);

  // residual of the pairs this thread finishes, fp32, for the whole call; their gates
  float2 res[TURNS], gate[TURNS];
#pragma unroll
  for (int t = 0; t < TURNS; ++t) {
    const int row = t * ROWS + e_row;
    res[t] = gate[t] = make_float2(0.f, 0.f);
    if (e_on && row < B)
      res[t] = rr::unpack(__ldg(reinterpret_cast<const unsigned int*>(p.embedding + token(row) * d + f0 + e_f)));
  }
  // ---- W_h h of a layer: needs nothing of this token ----
  float rec[TURNS][1][1][NT][4];
  uint32_t wh[1][KB][8];
  auto load_w_h = [&](int l) {
    if (l < L && p.layer[l].h_prev != nullptr) load_rows<KB>(wh, p.layer[l].w_h, f0, d, d, gq, k);
  };
  auto recur = [&](int l) {
#pragma unroll
    for (int t = 0; t < TURNS; ++t)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int u = 0; u < 4; ++u) rec[t][0][0][nt][u] = 0.f;
    if (l >= L || p.layer[l].h_prev == nullptr) return;
    const char* h = reinterpret_cast<const char*>(p.layer[l].h_prev);
#pragma unroll
    for (int t = 0; t < TURNS; ++t) {
      uint4 x[NT][KB];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) x[nt][kb] = __ldg(reinterpret_cast<const uint4*>(h + x_off[t][nt] + kb * 64));
      if (t == 0 && p.layer[l].scale != nullptr) {   // the normalised matrix, rounded as its copy would be
        const float scale = __ldg(p.layer[l].scale);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
          for (int j = 0; j < 8; ++j) wh[0][kb][j] = scaled(wh[0][kb][j], scale);
      }
      rr::products(rec[t], wh, x);
    }
  };
  auto load_bias = [&](int l) {
    return l < L && e_on ? rr::unpack(__ldg(reinterpret_cast<const unsigned int*>(p.layer[l].bias + f0 + e_f)))
                         : make_float2(0.f, 0.f);
  };
  load_w_h(0);
  recur(0);
  float2 bias = load_bias(0);
  settle_norm();
  __syncthreads();

  // the norm's output rows for layer l (l == L: the head)
  auto norm_input = [&](int l, int t, uint4 (&x)[NT][KB]) {
    if (l == 0) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const long long tok = token(min(t * ROWS + nt * 8 + gq, B - 1));
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          x[nt][kb] = __ldg(reinterpret_cast<const uint4*>(p.embedding + tok * d + k.col + kb * 32));
      }
    } else {
      const char* src = reinterpret_cast<const char*>(p.rb + (long)(l - 1) * B * d);
      rr::look(x, src, x_off[t]);
      if (!rr::await(x, src, x_off[t], l == p.stall_layer && blockIdx.x == 0, p.spin_limit, p.abort_word)) give_up(l);
      __syncwarp();
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float q = 0.f;
#pragma unroll
      for (int kb = 0; kb < KB; ++kb)
        if (k.owns(kb)) q += square_sum(x[nt][kb]);     // columns another warp counts: not here
      q += __shfl_xor_sync(0xffffffffu, q, 1);
      q += __shfl_xor_sync(0xffffffffu, q, 2);
      if (tq == 0) ss[nt * 8 + gq][warp] = q;
    }
    __syncthreads();
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const float4 q0 = *reinterpret_cast<const float4*>(&ss[nt * 8 + gq][0]);
      const float4 q1 = *reinterpret_cast<const float4*>(&ss[nt * 8 + gq][4]);
      const float rs = rsqrtf((((q0.x + q0.y) + (q0.z + q0.w)) + ((q1.x + q1.y) + (q1.z + q1.w))) / (float)d + p.eps);
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) {
        const uint4 n = *reinterpret_cast<const uint4*>(s_norm + (l & 1) * d + k.col + kb * 32);
        x[nt][kb].x = normed(x[nt][kb].x, n.x, rs); x[nt][kb].y = normed(x[nt][kb].y, n.y, rs);
        x[nt][kb].z = normed(x[nt][kb].z, n.z, rs); x[nt][kb].w = normed(x[nt][kb].w, n.w, rs);
      }
    }
  };

  for (int l = 0; l < L && !dead; ++l) {
    const long buf = (long)l * B * d;
    // ---- in_proj: the x and the z rows of my features ----
    await_rows(0, l);
#pragma unroll
    for (int t = 0; t < TURNS; ++t) {
      uint32_t w[1][KB][8];
      slot_rows(w, 0);
      uint4 x[NT][KB];
      norm_input(l, t, x);                   // (its barrier: nobody reads the partial sums any more)
      float acc[1][1][NT][4];
      rr::products(acc, w, x);
      put(0, acc);
      slot_rows(w, 1);
      rr::products(acc, w, x);
      put(1, acc);
      __syncthreads();
      if (s_bad[turn & 1]) { dead = true; break; }
      if (t + 1 == TURNS) send_for(0, l + 1);
      const int row = t * ROWS + e_row;
      if (e_on && row < B) {
        const float2 a = pair_total(0), z = pair_total(1);
        const float2 xr = rr::unpack(rr::pack(a.x, a.y)), zr = rr::unpack(rr::pack(z.x, z.y));
        store_pair(p.xa + buf, row, xr.x * rr::sigmoid_fast(xr.x), xr.y * rr::sigmoid_fast(xr.y));
        gate[t] = make_float2(zr.x * rr::sigmoid_fast(zr.x), zr.y * rr::sigmoid_fast(zr.y));
      }
      ++turn;
    }
    if (dead) break;
    stage_norm(l + 1);
    prefetch_w_h(l + 2);
    // ---- W_x x + W_h h + b, tanh, gate ----
    bf16* const h_out = p.layer[l].h_out;
    await_rows(1, l);
    {
      uint32_t w[1][KB][8];
      slot_rows(w, 2);
#pragma unroll
      for (int t = 0; t < TURNS; ++t) {
        uint4 x[NT][KB];
        const char* src = reinterpret_cast<const char*>(p.xa + buf);
          rr::look(x, src, x_off[t]);
        if (!rr::await(x, src, x_off[t], false, p.spin_limit, p.abort_word)) give_up(l);
        __syncwarp();
        float acc[1][1][NT][4];
        rr::products(acc, w, x);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int u = 0; u < 4; ++u) acc[0][0][nt][u] += rec[t][0][0][nt][u];
        settle_norm();
        __syncthreads();                     // nobody reads the partial sums any more
        put(0, acc);
        __syncthreads();
        if (s_bad[turn & 1]) { dead = true; break; }
        if (t + 1 == TURNS) send_for(1, l + 1);
        const int row = t * ROWS + e_row;
        if (e_on && row < B) {
          const float2 a = pair_total(0);
          const float h0 = rr::tanh_fast(a.x + bias.x), h1 = rr::tanh_fast(a.y + bias.y);
          store_pair(p.y + buf, row, h0 * gate[t].x, h1 * gate[t].y);
          *reinterpret_cast<uint32_t*>(h_out + (long)row * d + f0 + e_f) = rr::pack(h0, h1);
        }
        ++turn;
      }
    }
    if (dead) break;
    // ---- out_proj, residual; the next layer's W_h h while y is on its way ----
    bias = load_bias(l + 1);
    load_w_h(l + 1);
    recur(l + 1);
    await_rows(2, l);
    {
      uint32_t w[1][KB][8];
      slot_rows(w, 3);
#pragma unroll
      for (int t = 0; t < TURNS; ++t) {
        uint4 x[NT][KB];
        const char* src = reinterpret_cast<const char*>(p.y + buf);
          rr::look(x, src, x_off[t]);
        if (!rr::await(x, src, x_off[t], false, p.spin_limit, p.abort_word)) give_up(l);
        __syncwarp();
        float acc[1][1][NT][4];
        rr::products(acc, w, x);
        __syncthreads();
        put(0, acc);
        __syncthreads();
        if (s_bad[turn & 1]) { dead = true; break; }
        if (t + 1 == TURNS) send_for(2, l + 1);
        const int row = t * ROWS + e_row;
        if (e_on && row < B) {
          const float2 a = pair_total(0), o = rr::unpack(rr::pack(a.x, a.y));
          res[t].x += o.x; res[t].y += o.y;
          store_pair(p.rb + buf, row, res[t].x, res[t].y);
        }
        ++turn;
      }
    }
  }
  if (dead) {
    // Nothing may still be landing in this CTA's shared memory when it goes: the rows sent for last
    // (a group's earlier ones had landed before these were sent for).  They come from this device's
    // own memory and always arrive; the wait's time limit is its bound.
    settle_norm();
    __syncthreads();
    land(landed, s_sent);
    __syncthreads();
    return;
  }

  // ---- final norm and head: units of 16 vocabulary rows ----
  for (int v0 = blockIdx.x * LT_R; v0 < p.V; v0 += gridDim.x * LT_R) {
    load_rows<KB>(wh, p.head, v0, p.V, d, gq, k);
#pragma unroll
    for (int t = 0; t < TURNS; ++t) {
      uint4 x[NT][KB];
      norm_input(L, t, x);
      float acc[1][1][NT][4];
      rr::products(acc, wh, x);
      put(0, acc);
      __syncthreads();
      if (s_bad[turn & 1]) return;
      const int row = t * ROWS + e_row;
      if (tid < ROWS * 8 && row < B) {
        const float2 a = pair_total(0);
        bf16* out = p.logits + (long)row * p.V + v0 + e_f;
        if (v0 + e_f < p.V) out[0] = __float2bfloat16_rn(a.x);
        if (v0 + e_f + 1 < p.V) out[1] = __float2bfloat16_rn(a.y);
      }
      ++turn;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Power iteration of several matrices: v = W^T u / (|W^T u| + eps), u = W v / (|W v| + eps), three
// times, then scale = target / (|u^T W v| + eps) (elman/models/mamba_gated_elman.py:123-146).
// NC CTAs per matrix own R = ceil(d / NC) rows of W (and as many columns of v) and keep the rows in
// shared memory.  Two hand-offs per iteration: every CTA's partial of W^T u to the owners of its
// columns, the sums back to all.  u is passed on unnormalised; its norm travels with the partials.
// ---------------------------------------------------------------------------------------------
constexpr int SP_THREADS = 512;
constexpr int SP_ITERS = 3;
constexpr int SP_MAX_NC = 64;

struct SpectralManyParams {
  int d, NC, R, groups;            // groups: row groups of the column pass
  float target, eps;
  float* exchange;                 // per matrix: [ITERS][NC][d] partials, [ITERS][d] sums, [ITERS + 1][NC] squares
  long exchange_stride;
  int* abort_word;
  int* status;
  long spin_limit;
  int stall_iter;                  // test hook: block 0 waits in this iteration for what never comes (-1 off)
  const bf16* W[LT_MAX_LAYERS];
  bf16* u[LT_MAX_LAYERS];
  float* scale[LT_MAX_LAYERS];
};

__host__ __device__ inline long spectral_exchange_floats(int d, int NC) {
  return ((long)SP_ITERS * (NC + 1) * d + (SP_ITERS + 1) * NC + 63) / 64 * 64;
}

// Words from other CTAs, when they are there: N at a time, all in flight (at(i) null: none).
template <int N, typename At>
__device__ __forceinline__ void await_words(float (&v)[N], At at, const SpectralManyParams& p, int* bad) {
  uint32_t w[N];
#pragma unroll
  for (int i = 0; i < N; ++i) w[i] = 0xFFFFFFFFu;
  long spins = 0;
  unsigned long long t_begin = 0;
  while (true) {
    bool pending = false;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (w[i] == 0xFFFFFFFFu) {
        const float* a = at(i);
        w[i] = 0u;
        if (a != nullptr) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w[i]) : "l"(a) : "memory");
      }
#pragma unroll
    for (int i = 0; i < N; ++i) pending = pending || w[i] == 0xFFFFFFFFu;
    if (!pending) break;
    bool stop = ++spins > p.spin_limit;
    if ((spins & 63) == 0) {
      const unsigned long long now = ptx::globaltimer_ns();
      if (t_begin == 0) t_begin = now;
      stop = stop || ld_relaxed_gpu(p.abort_word) == 1 || now - t_begin > ptx::kWaitDeadlineNs;
    }
    if (stop) {
      if (atomicExch(p.abort_word, 1) != 1) report_timeout(p.status, KID_LM_TOKEN, 0xFFFF);
      *bad = 1;
      break;
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = __uint_as_float(w[i]);
}

// STALL: with the test hook (its one comparison cost 0.6 of 25 us).
template <bool STALL>
__global__ void __launch_bounds__(SP_THREADS, 1) spectral_many_kernel(const __grid_constant__ SpectralManyParams p) {
  extern __shared__ __align__(16) float sp_smem[];
  __shared__ float s_red[SP_THREADS / 32];
  __shared__ float s_sq[SP_MAX_NC];
  __shared__ __align__(8) uint64_t landed;
  __shared__ int s_bad;
  const int d = p.d, NC = p.NC, R = p.R;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int mat = blockIdx.x / NC, c = blockIdx.x - mat * NC;
  const int r0 = c * R, rows = max(0, min(R, d - r0));      // my rows of W = my columns of v
  float* t = sp_smem;                       // [d]           W^T u
  float* red = t + d;                       // [groups][d]   row groups of the column pass
  float* stage = red + p.groups * d;        // [NC][R]       partials of my columns
  float* u = stage + (NC * R + 3) / 4 * 4;  // [R]           my rows of u, unnormalised
  bf16* W = reinterpret_cast<bf16*>(u + (R + 3) / 4 * 4);   // [R][d], on a 16-byte boundary
  float* ex = p.exchange + mat * p.exchange_stride;
  float* ex_sum = ex + (long)SP_ITERS * NC * d;
  float* ex_sq = ex_sum + (long)SP_ITERS * d;
  if (tid == 0) {
    ptx::mbar_init(&landed, 1);
    ptx::mbar_fence_init();
    s_bad = 0;
    if (rows > 0) {     // my rows are one piece of memory: one bulk copy
      const uint32_t bytes = (uint32_t)(rows * d) * 2u;
      ptx::mbar_arrive_expect_tx(&landed, bytes);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(ptx::smem_u32(W)), "l"(p.W[mat] + (long)r0 * d), "r"(bytes), "r"(ptx::smem_u32(&landed))
                   : "memory");
    }
  }
  for (int r = tid; r < rows; r += SP_THREADS) u[r] = __bfloat162float(p.u[mat][r0 + r]);
  __syncthreads();
  if (rows > 0) {
    // (the copy is local to this device and always ends; the limit is the status word's)
    int none = 0;
    if (!ptx::mbar_wait(&landed, 0, 1L << 40, &none)) return;
  }
  auto block_sum = [&](float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) s_red[warp] = x;
    __syncthreads();
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < SP_THREADS / 32; ++w) v += s_red[w];
    __syncthreads();
    return v;
  };
  const int c8 = d / 8, cg = tid / c8, cc = tid - cg * c8;   // column pass: row group, column octet
  float inv_u = 1.f, norm_u = 0.f;
  for (int it = 0; it < SP_ITERS; ++it) {
    // ---- my rows' part of W^T u ----
    if (cg < p.groups) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int r = cg; r < rows; r += p.groups) {
        const uint4 q = *reinterpret_cast<const uint4*>(W + (long)r * d + cc * 8);
        const float2 a = rr::unpack(q.x), b = rr::unpack(q.y), e = rr::unpack(q.z), f = rr::unpack(q.w);
        const float ur = u[r];
        acc[0] += a.x * ur; acc[1] += a.y * ur; acc[2] += b.x * ur; acc[3] += b.y * ur;
        acc[4] += e.x * ur; acc[5] += e.y * ur; acc[6] += f.x * ur; acc[7] += f.y * ur;
      }
#pragma unroll
      for (int j = 0; j < 8; j += 4)
        *reinterpret_cast<float4*>(red + cg * d + cc * 8 + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
    }
    __syncthreads();
    float* mine = ex + ((long)it * NC + c) * d;
    for (int col = tid; col < d; col += SP_THREADS) {
      float v = 0.f;
      for (int g = 0; g < p.groups; ++g) v += red[g * d + col];
      rr::st_relaxed_u32(mine + col, __float_as_uint(v));
    }
    // ---- my columns: everybody's partials, and the norm of the u they came from ----
    if (STALL && it == p.stall_iter && blockIdx.x == 0 && tid == 0) {   // (no square sums come before iteration 1)
      float v[1];
      await_words<1>(v, [&](int) { return ex_sq; }, p, &s_bad);
    }
    constexpr int NW = 4;
    for (int e0 = tid; e0 < NC * rows; e0 += NW * SP_THREADS) {
      float v[NW];
      await_words<NW>(v, [&](int i) -> const float* {
        const int e = e0 + i * SP_THREADS, q = e / rows;
        return e < NC * rows ? ex + ((long)it * NC + q) * d + r0 + e - q * rows : nullptr;
      }, p, &s_bad);
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        const int e = e0 + i * SP_THREADS, q = e / rows;
        if (e < NC * rows) stage[q * R + e - q * rows] = v[i];
      }
    }
    if (it > 0 && tid < NC) {
      float v[1];
      await_words<1>(v, [&](int) { return ex_sq + it * NC + tid; }, p, &s_bad);
      s_sq[tid] = v[0];
    }
    __syncthreads();
    if (s_bad) return;
    if (it > 0) {
      float nu = 0.f;
      for (int q = 0; q < NC; ++q) nu += s_sq[q];
      inv_u = 1.f / (sqrtf(nu) + p.eps);
    }
    for (int j = tid; j < rows; j += SP_THREADS) {
      float v = 0.f;
      for (int q = 0; q < NC; ++q) v += stage[q * R + j];
      rr::st_relaxed_u32(ex_sum + it * d + r0 + j, __float_as_uint(v * inv_u));
    }
    // ---- all of W^T u, its norm ----
    float sq = 0.f;
    for (int c0 = tid; c0 < d; c0 += NW * SP_THREADS) {
      float v[NW];
      await_words<NW>(v, [&](int i) -> const float* {
        return c0 + i * SP_THREADS < d ? ex_sum + it * d + c0 + i * SP_THREADS : nullptr;
      }, p, &s_bad);
#pragma unroll
      for (int i = 0; i < NW; ++i)
        if (c0 + i * SP_THREADS < d) { t[c0 + i * SP_THREADS] = v[i]; sq += v[i] * v[i]; }
    }
    const float inv_v = 1.f / (sqrtf(block_sum(sq)) + p.eps);
    if (s_bad) return;
    // ---- my rows of W v ----
    sq = 0.f;
    constexpr int RI = 4;                    // rows in flight per warp: they share the reads of t
    for (int rb = warp * RI; rb < rows; rb += SP_THREADS / 32 * RI) {
      float acc[RI];
#pragma unroll
      for (int i = 0; i < RI; ++i) acc[i] = 0.f;
      for (int col = lane * 8; col < d; col += 256) {
        const float4 t0 = *reinterpret_cast<const float4*>(t + col), t1 = *reinterpret_cast<const float4*>(t + col + 4);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          const uint4 q = *reinterpret_cast<const uint4*>(W + (long)min(rb + i, rows - 1) * d + col);
          const float2 a = rr::unpack(q.x), b = rr::unpack(q.y), e = rr::unpack(q.z), f = rr::unpack(q.w);
          acc[i] += a.x * t0.x + a.y * t0.y + b.x * t0.z + b.y * t0.w + e.x * t1.x + e.y * t1.y + f.x * t1.z + f.y * t1.w;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < RI; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        const float w = acc[i] * inv_v;
        if (lane == 0 && rb + i < rows) { u[rb + i] = w; sq += w * w; }
      }
    }
    sq = block_sum(sq);
    if (tid == 0) rr::st_relaxed_u32(ex_sq + (it + 1) * NC + c, __float_as_uint(sq));
  }
  if (tid < NC) {
    float v[1];
    await_words<1>(v, [&](int) { return ex_sq + SP_ITERS * NC + tid; }, p, &s_bad);
    s_sq[tid] = v[0];
  }
  __syncthreads();
  if (s_bad) return;
  float nu = 0.f;
  for (int q = 0; q < NC; ++q) nu += s_sq[q];
  norm_u = sqrtf(nu);
  inv_u = 1.f / (norm_u + p.eps);
  for (int r = tid; r < rows; r += SP_THREADS) p.u[mat][r0 + r] = __float2bfloat16_rn(u[r] * inv_u);
  // |u^T W v| with u = W v / (|W v| + eps)
  if (c == 0 && tid == 0) *p.scale[mat] = p.target / (fabsf(norm_u * norm_u * inv_u) + p.eps);
}

// How many matrices go through one launch, and on how many CTAs each.
struct SpectralPlan { int per_launch, NC, R, groups; size_t smem; };
bool spectral_plan(int L, int d, SpectralPlan* out) {
  for (int m = L; m >= 1; --m) {
    int NC = rec_reg_sms() / m;
    if (NC > SP_MAX_NC) NC = SP_MAX_NC;
    if (NC > d / 8) NC = d / 8;
    const int R = (d + NC - 1) / NC;
    int groups = SP_THREADS / (d / 8);
    if (groups > 16) groups = 16;
    if (groups < 1) return false;
    const size_t smem = ((size_t)d + (size_t)groups * d + (NC * R + 3) / 4 * 4 + (R + 3) / 4 * 4) * 4 +
                        (size_t)R * d * 2;
    if (smem > SP_SMEM_LIMIT) continue;
    *out = {m, NC, R, groups, smem};
    return true;
  }
  return false;
}

typedef void (*LmTokenKernel)(const LmTokenParams);
// Sequences in turns of at most 32: all of a turn's looks are in flight together.
int token_tiles(int B) { return B <= 8 ? 1 : B <= 16 ? 2 : 4; }
template <int KB>
LmTokenKernel by_tiles(int B) {
  return B <= 8 ? lm_token_kernel<KB, 1, 1> : B <= 16 ? lm_token_kernel<KB, 2, 1>
         : B <= 32 ? lm_token_kernel<KB, 4, 1> : lm_token_kernel<KB, 4, 2>;
}
LmTokenKernel pick_token_kernel(int d, int B) {
  switch (((d + 31) / 32 + RR_WARPS - 1) / RR_WARPS) {
    case 1: return by_tiles<1>(B);
    case 2: return by_tiles<2>(B);
    case 3: return by_tiles<3>(B);
    case 4: return by_tiles<4>(B);
    case 5: return by_tiles<5>(B);
    case 6: return by_tiles<6>(B);
  }
  return nullptr;
}

// Behind a power iteration, which has advanced its vectors, nothing may start over.
int too_late(int rc) {
  return rc != ELMAN_ERR_UNSUPPORTED
             ? rc : set_error(ELMAN_ERR_CUDA, "a cooperative launch was refused behind the power iterations");
}

size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

}  // namespace

bool lm_token_supported(int dtype, int L, int B, int d, int V) {
  if (dtype != ELMAN_BF16 || options().force_generic != 0 || options().rec_reg == 1) return false;
  if (L < 1 || L > LT_MAX_LAYERS || B < 1 || B > LT_MAX_ROWS || V < 1) return false;
  SpectralPlan sp;
  return d >= 32 && (d & 7) == 0 && d <= 1536 && (d + LT_R - 1) / LT_R <= rec_reg_sms() &&
         lt_smem(d, token_tiles(B)) <= LT_SMEM_LIMIT && spectral_plan(L, d, &sp);
}

// Everything that starts out as "not there yet", in one piece: three activation buffers per layer,
// the power iterations' exchange, the abort word; then the scales.
size_t lm_token_workspace(int L, int B, int d) {
  SpectralPlan sp;
  if (d < 32 || !spectral_plan(L, d, &sp)) return 256;
  return align256((size_t)3 * L * B * d * sizeof(bf16)) +
         align256((size_t)L * spectral_exchange_floats(d, sp.NC) * sizeof(float)) + 256 +
         align256((size_t)L * sizeof(float));
}

int lm_token(const LmTokenArgs& a, cudaStream_t stream) {
  SpectralPlan sp;
  if (!spectral_plan(a.L, a.d, &sp)) return ELMAN_ERR_UNSUPPORTED;
  const size_t act = align256((size_t)3 * a.L * a.B * a.d * sizeof(bf16));
  const long ex_floats = spectral_exchange_floats(a.d, sp.NC);
  const size_t exb = align256((size_t)a.L * ex_floats * sizeof(float));
  char* ws = (char*)a.workspace;
  LmTokenParams p{};
  SpectralManyParams q{};
  p.L = a.L; p.B = a.B; p.d = a.d; p.V = a.V;
  p.tokens = a.tokens;
  p.embedding = (const bf16*)a.embedding; p.norm = (const bf16*)a.norm; p.head = (const bf16*)a.head;
  p.eps = a.eps;
  p.rb = (bf16*)ws;
  p.xa = p.rb + (size_t)a.L * a.B * a.d;
  p.y = p.xa + (size_t)a.L * a.B * a.d;
  p.logits = (bf16*)a.logits;
  p.abort_word = (int*)(ws + act + exb);
  float* scales = (float*)(ws + act + exb + 256);
  p.status = device_status_ptr();
  p.spin_limit = options().spin_limit;
  const long stall = options().test_stall_step;     // a layer, or 1000 + an iteration of the power iterations
  p.stall_layer = stall < 1000 ? (int)stall : -1;
  q.stall_iter = stall < 1000 ? -1 : (int)(stall - 1000);
  // read 16 bytes at a time; in feature pairs
  uintptr_t wide = (uintptr_t)a.embedding | (uintptr_t)a.norm | (uintptr_t)a.head | (uintptr_t)ws;
  uintptr_t narrow = 0;
  q.d = a.d; q.NC = sp.NC; q.R = sp.R; q.groups = sp.groups;
  q.target = a.target; q.eps = a.spectral_eps;
  q.exchange_stride = ex_floats;
  q.abort_word = p.abort_word; q.status = p.status; q.spin_limit = p.spin_limit;
  int normed[LT_MAX_LAYERS], n_normed = 0;
  for (int l = 0; l < a.L; ++l) {
    const void* const* r = a.layers + (size_t)l * LM_TOKEN_REFS;
    LayerRefs& o = p.layer[l];
    o.norm = (const bf16*)r[0]; o.w_in = (const bf16*)r[1]; o.w_x = (const bf16*)r[2];
    o.w_h = (const bf16*)r[3]; o.bias = (const bf16*)r[4]; o.w_out = (const bf16*)r[5];
    o.h_prev = (const bf16*)r[7]; o.h_out = (bf16*)r[8];
    for (int k = 0; k < 6; ++k)
      if (r[k] == nullptr) return set_error(ELMAN_ERR_ARG, "layer %d: pointer %d is NULL", l, k);
    if (r[8] == nullptr) return set_error(ELMAN_ERR_ARG, "layer %d: pointer 8 is NULL", l);
    wide |= (uintptr_t)r[0] | (uintptr_t)r[1] | (uintptr_t)r[2] | (uintptr_t)r[3] | (uintptr_t)r[5] | (uintptr_t)r[7];
    narrow |= (uintptr_t)r[4] | (uintptr_t)r[8];
    o.scale = r[6] != nullptr ? scales + l : nullptr;
    if (r[6] != nullptr) normed[n_normed++] = l;
  }
  if ((wide & 15) != 0 || (narrow & 3) != 0) return ELMAN_ERR_UNSUPPORTED;
  LmTokenKernel kern = pick_token_kernel(a.d, a.B);
  if (kern == nullptr) return ELMAN_ERR_UNSUPPORTED;
  cudaLaunchConfig_t cfg{}, sp_cfg{};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;   // the CTAs of either launch wait for one another
  attr.val.cooperative = 1;
  cfg.attrs = sp_cfg.attrs = &attr;
  cfg.numAttrs = sp_cfg.numAttrs = 1;
  cfg.stream = sp_cfg.stream = stream;
  cfg.gridDim = dim3((a.d + LT_R - 1) / LT_R);
  cfg.blockDim = dim3(LT_THREADS);
  cfg.dynamicSmemBytes = lt_smem(a.d, token_tiles(a.B));
  sp_cfg.gridDim = dim3((n_normed < sp.per_launch ? n_normed : sp.per_launch) * sp.NC);
  sp_cfg.blockDim = dim3(SP_THREADS);
  sp_cfg.dynamicSmemBytes = sp.smem;
  void (*const power)(const SpectralManyParams) = q.stall_iter < 0 ? spectral_many_kernel<false> : spectral_many_kernel<true>;
  ELMAN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM_LIMIT));
  if (!fits_together((const void*)kern, cfg)) return ELMAN_ERR_UNSUPPORTED;
  if (n_normed > 0) {
    ELMAN_CUDA_CHECK(cudaFuncSetAttribute(power, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          SP_SMEM_LIMIT));
    if (!fits_together((const void*)power, sp_cfg)) return ELMAN_ERR_UNSUPPORTED;
  }
  ELMAN_CUDA_CHECK(cudaMemsetAsync(ws, 0xFF, act + exb + 256, stream));
  for (int i = 0; i < n_normed; i += sp.per_launch) {
    const int m = n_normed - i < sp.per_launch ? n_normed - i : sp.per_launch;
    for (int j = 0; j < m; ++j) {
      const void* const* r = a.layers + (size_t)normed[i + j] * LM_TOKEN_REFS;
      q.W[j] = (const bf16*)r[3]; q.u[j] = (bf16*)const_cast<void*>(r[6]); q.scale[j] = scales + normed[i + j];
    }
    q.exchange = (float*)(ws + act) + (size_t)i * ex_floats;
    sp_cfg.gridDim = dim3(m * sp.NC);
    const int rc = launch_together(power, sp_cfg, q);
    if (rc != ELMAN_OK) return i == 0 ? rc : too_late(rc);
    count_launch(false);
  }
  const int rc = launch_together(kern, cfg, p);
  if (rc != ELMAN_OK) return n_normed == 0 ? rc : too_late(rc);
  count_launch(true);
  return ELMAN_OK;
}

}  // namespace elman
