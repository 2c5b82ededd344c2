// Dense recurrence in single precision with the recurrent matrix in registers.
//
// The chain of rec_reg.cuh — batch groups, K split over eight warps, the state tensor filled with a
// pattern (0xFFFFFFFF, a NaN no arithmetic produces) as its own message, one store and one load
// through L2 per step — around FFMA: lane l of every warp owns row l of the CTA's 32 rows of W and
// keeps that row's part of the warp's K range in registers (KW values).  A warp stages the four
// batch rows of its K range in shared memory, where every lane reads the same four values at a
// time.  Arithmetic is that of the cooperative kernel in rec_simt.cu (fp32 products and sums, tanhf).
//
// Bound by the hand-off: at B = 4, d = 256 a step is 0.26 M multiply-adds on 8 CTAs, 128 per lane.
// Measured (us per step forward / backward, against the cooperative kernel):
//    B = 4,  d = 256   4.72  4.64 -> 0.90 0.87
//    B = 16, d = 512  13.8  12.8  -> 1.40 1.40
// (elman/cuda/lib/mamba_gated_elman_gpu.cu.cc:451-473, :527-558 of the reference)
#include "rec_reg.cuh"

namespace elman {

namespace {

constexpr int F32_R = 32;      // rows of W per CTA: one per lane
constexpr int F32_NG = 4;      // batch rows per group
constexpr int F32_MAX_KW = 128;

struct RecF32Params {
  int T, B, d;
  int b_lo, b_hi;         // batch rows of this launch
  int cpg;                // CTAs per batch group
  const float* W;         // row = output feature (backward: the transposed matrix)
  const float* in0;       // forward pre            backward g
  const float* in1;       // forward g              backward dy
  const float* in2;       //                        backward h [T+1 slots]
  const float* in3;       //                        backward v
  float* state;           // forward h [T+1 slots]  backward dv [T+1 slots]
  float* out0;            // forward v (or null)    backward dg (or null)
  float* out1;            // forward y
  float* db;
  int* abort_word;
  int* status;
  long spin_limit;
  int self_gate;
  int stall_step;         // test hook: block 0 never sees its input of this step (-1 off)
};

template <bool BWD, int KW>
__global__ void __launch_bounds__(RR_THREADS, 1) rec_f32_kernel(const RecF32Params p) {
  constexpr int R = F32_R, NG = F32_NG, Q4 = KW / 4;
  constexpr int LOOKS = (NG * Q4 + 31) / 32;     // 16-byte pieces of state per lane
  constexpr int XS = KW + 4;
  constexpr int NIN = BWD ? 4 : 2;
  __shared__ __align__(16) float xs[RR_WARPS][NG][XS];
  __shared__ float part[2][RR_WARPS][NG][R];
  __shared__ float ring[RR_AHEAD][NIN][R * NG];
  __shared__ int s_bad[2];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = p.T, d = p.d;
  const int grp = blockIdx.x / p.cpg, c = blockIdx.x - grp * p.cpg;
  const int f0 = c * R, b0 = p.b_lo + grp * NG;
  const int k0 = warp * KW;
  if (tid < 2) s_bad[tid] = 0;

  float w[KW];
#pragma unroll
  for (int k = 0; k < KW; k += 4) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (f0 + lane < d && k0 + k < d)
      x = __ldg(reinterpret_cast<const float4*>(p.W + (long)(f0 + lane) * d + k0 + k));
    w[k] = x.x; w[k + 1] = x.y; w[k + 2] = x.z; w[k + 3] = x.w;
  }
  // the pieces of state this lane looks for: batch row n, columns k0 + 4 k4 ..
  uint32_t x_off[1][LOOKS];
  float* x_to[LOOKS];
  bool x_on[LOOKS];
#pragma unroll
  for (int j = 0; j < LOOKS; ++j) {
    const int q = lane + 32 * j, n = q / Q4, k4 = q - n * Q4;
    x_on[j] = n < NG && k0 + 4 * k4 < d;
    // a row past the batch reads the last row's state: its products are discarded
    x_off[0][j] = x_on[j] ? (uint32_t)(min(b0 + n, p.b_hi - 1) * d + k0 + 4 * k4) * 4u : 0u;
    x_to[j] = &xs[warp][n < NG ? n : 0][4 * k4];
    if (n < NG && !x_on[j]) *reinterpret_cast<float4*>(x_to[j]) = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  // the element this thread finishes
  const int n_e = tid / R, f_e = tid - n_e * R;
  const bool mine = tid < R * NG && f0 + f_e < d && b0 + n_e < p.b_hi;
  const uint32_t off = mine ? (uint32_t)((b0 + n_e) * d + f0 + f_e) * 4u : 0u;
  const int slot = p.B * d * 4;
  auto word = [](const float* base, long at, uint32_t off) {
    return reinterpret_cast<const unsigned int*>(reinterpret_cast<const char*>(base) + at + off);
  };
  auto fetch = [&](int s, long at) {
    if (s < T && mine) {
      uint32_t* to = reinterpret_cast<uint32_t*>(&ring[s & (RR_AHEAD - 1)][0][tid]);
      rr::copy_word(to, word(p.in0, at, off));
      if (BWD || !p.self_gate) rr::copy_word(to + R * NG, word(p.in1, at, off));
      if (BWD) {
        rr::copy_word(to + 2 * R * NG, word(p.in2, at + slot, off));
        rr::copy_word(to + 3 * R * NG, word(p.in3, at, off));
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const long step_bytes = BWD ? -(long)slot : (long)slot;
  long at = BWD ? (long)(T - 1) * slot : 0;
#pragma unroll
  for (int s = 0; s < RR_AHEAD - 1; ++s) fetch(s, at + s * step_bytes);
  float db_acc = 0.f;
  const int stall_step = blockIdx.x == 0 ? p.stall_step : -1;
  __syncthreads();

  for (int s = 0; s < T; ++s, at += step_bytes) {
    // ---- step-local arithmetic: forward e0 = pre, e1 = silu(g); backward e0 = dy * gate term,
    // e1 = 1 - tanh(v)^2, late = dg ----
    fetch(s + RR_AHEAD - 1, at + (RR_AHEAD - 1) * step_bytes);
    asm volatile("cp.async.wait_group %0;" ::"n"(RR_AHEAD - 1) : "memory");
    float e0 = 0.f, e1 = 0.f, late = 0.f;
    if (mine) {
      const float* in = &ring[s & (RR_AHEAD - 1)][0][tid];
      if (!BWD) {
        e0 = in[0];
        if (!p.self_gate) e1 = siluf_(in[R * NG]);
      } else {
        const float dy = in[R * NG], h = in[(NIN - 2) * R * NG], th = tanhf(in[(NIN - 1) * R * NG]);
        if (!p.self_gate) {
          const float g = in[0];
          e0 = dy * siluf_(g);
          late = dy * h * dsiluf_(g);
        } else {   // y = h silu(h): d y / d h = silu(h) + h silu'(h)
          e0 = dy * (siluf_(h) + h * dsiluf_(h));
        }
        e1 = 1.f - th * th;
      }
    }
    asm volatile("" : "+f"(e0), "+f"(e1), "+f"(late));
    // ---- the group's state over my K range, into shared memory as it arrives ----
    const char* src = reinterpret_cast<const char*>(p.state) + (BWD ? at + slot : at);
    uint4 x[LOOKS];
    long spins = 0;
    unsigned long long t_begin = 0;
#pragma unroll
    for (int j = 0; j < LOOKS; ++j) x[j] = rr::ld_relaxed_v4(src + x_off[0][j]);
    while (s > 0) {
      uint32_t top = s == stall_step ? 0xFFFFFFFFu : 0u;
#pragma unroll
      for (int j = 0; j < LOOKS; ++j) top = max(top, x_on[j] ? rr::largest(x[j]) : 0u);
      if (top != 0xFFFFFFFFu) break;
#pragma unroll
      for (int j = 0; j < LOOKS; ++j)
        if (x_on[j] && rr::largest(x[j]) == 0xFFFFFFFFu) x[j] = rr::ld_relaxed_v4(src + x_off[0][j]);
      bool stop = ++spins > p.spin_limit;
      if ((spins & 63) == 0) {
        const unsigned long long now = ptx::globaltimer_ns();
        if (t_begin == 0) t_begin = now;
        stop = stop || ld_relaxed_gpu(p.abort_word) != 0 || now - t_begin > ptx::kWaitDeadlineNs;
      }
      if (stop) {
        if (atomicExch(p.abort_word, 1) == 0) report_timeout(p.status, KID_REC_SIMT, s);
        s_bad[s & 1] = 1;
        break;
      }
    }
    __syncwarp();          // the last step's reads of xs are done
#pragma unroll
    for (int j = 0; j < LOOKS; ++j)
      if (x_on[j])
        *reinterpret_cast<uint4*>(x_to[j]) = x[j];
    __syncwarp();
    float acc[NG];
#pragma unroll
    for (int n = 0; n < NG; ++n) acc[n] = 0.f;
#pragma unroll
    for (int k = 0; k < KW; k += 4)
#pragma unroll
      for (int n = 0; n < NG; ++n) {
        const float4 v = *reinterpret_cast<const float4*>(&xs[warp][n][k]);
        acc[n] = fmaf(w[k], v.x, acc[n]);
        acc[n] = fmaf(w[k + 1], v.y, acc[n]);
        acc[n] = fmaf(w[k + 2], v.z, acc[n]);
        acc[n] = fmaf(w[k + 3], v.w, acc[n]);
      }
#pragma unroll
    for (int n = 0; n < NG; ++n) part[s & 1][warp][n][lane] = acc[n];
    __syncthreads();
    const int bad = s_bad[s & 1];
    if (mine) {
      float a = 0.f;
#pragma unroll
      for (int wv = 0; wv < RR_WARPS; ++wv) a += part[s & 1][wv][n_e][f_e];
      char* dst = reinterpret_cast<char*>(p.state) + (BWD ? at : at + slot) + off;
      if (!BWD) {
        a += e0;
        const float h = tanhf(a);
        rr::st_relaxed_u32(dst, __float_as_uint(h));
        if (p.out0 != nullptr) *const_cast<unsigned int*>(word(p.out0, at, off)) = __float_as_uint(a);
        *const_cast<unsigned int*>(word(p.out1, at, off)) =
            __float_as_uint(h * (p.self_gate ? siluf_(h) : e1));
      } else {
        const float dv = (e0 + a) * e1;
        rr::st_relaxed_u32(dst, __float_as_uint(dv));
        db_acc += dv;
        if (p.out0 != nullptr) *const_cast<unsigned int*>(word(p.out0, at, off)) = __float_as_uint(late);
      }
    }
    if (bad) break;
  }
  if (BWD) {   // bias gradient: the group's rows of a feature, in a fixed order
    __syncthreads();
    if (tid < R * NG) part[0][0][n_e][f_e] = db_acc;
    __syncthreads();
    if (tid < R && f0 + tid < d) {
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < NG; ++n) sum += part[0][0][n][tid];
      p.db[(long)(p.b_lo / NG + grp) * d + f0 + tid] = sum;
    }
  }
}

typedef void (*RecF32Kernel)(const RecF32Params);
template <bool BWD>
RecF32Kernel pick_f32(int kw) {
  if (kw <= 8) return rec_f32_kernel<BWD, 8>;
  if (kw <= 16) return rec_f32_kernel<BWD, 16>;
  if (kw <= 24) return rec_f32_kernel<BWD, 24>;
  if (kw <= 32) return rec_f32_kernel<BWD, 32>;
  if (kw <= 40) return rec_f32_kernel<BWD, 40>;
  if (kw <= 48) return rec_f32_kernel<BWD, 48>;
  if (kw <= 64) return rec_f32_kernel<BWD, 64>;
  if (kw <= 96) return rec_f32_kernel<BWD, 96>;
  return rec_f32_kernel<BWD, 128>;
}

// Groups that do not fit on the device together go through in slices: sequences are independent.
int f32_launch(bool bwd, RecF32Params& p, int* sync, cudaStream_t stream) {
  const uintptr_t wide = (uintptr_t)p.W | (uintptr_t)p.state;
  if ((wide & 15) != 0) return ELMAN_ERR_UNSUPPORTED;
  const int kw = (p.d + RR_WARPS - 1) / RR_WARPS;
  RecF32Kernel kern = bwd ? pick_f32<true>(kw) : pick_f32<false>(kw);
  p.cpg = (p.d + F32_R - 1) / F32_R;
  const int groups = (p.B + F32_NG - 1) / F32_NG, fit = rec_reg_sms() / p.cpg;
  if (fit < 1 || groups > REC_MAX_DB_ROWS) return ELMAN_ERR_UNSUPPORTED;
  const int launches = (groups + fit - 1) / fit, per = (groups + launches - 1) / launches;
  p.abort_word = sync;
  p.status = device_status_ptr();
  p.spin_limit = options().spin_limit;
  p.stall_step = (int)options().test_stall_step;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((per < groups ? per : groups) * p.cpg);
  cfg.blockDim = dim3(RR_THREADS);
  cfg.stream = stream;
  // the runtime's guarantee that the CTAs, which wait for one another, are resident together
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (!fits_together((const void*)kern, cfg)) return ELMAN_ERR_UNSUPPORTED;
  const size_t slot = (size_t)p.B * p.d * sizeof(float);
  ELMAN_CUDA_CHECK(cudaMemsetAsync(sync, 0, 4, stream));
  ELMAN_CUDA_CHECK(cudaMemsetAsync((char*)p.state + (bwd ? 0 : slot), 0xFF, (size_t)p.T * slot, stream));
  for (int g = 0; g < groups; g += per) {
    p.b_lo = g * F32_NG;
    p.b_hi = (g + per) * F32_NG < p.B ? (g + per) * F32_NG : p.B;
    cfg.gridDim = dim3((p.b_hi - p.b_lo + F32_NG - 1) / F32_NG * p.cpg);
    ELMAN_RETURN_IF(launch_together(kern, cfg, p));
    count_launch(false, REC_KERNEL_F32);
  }
  if (bwd && groups > 1) return fold_db_rows(p.db, p.d, groups, stream);
  return ELMAN_OK;
}

}  // namespace

// From 8 features up, 16-byte rows, at most 128 columns of a row per lane; the rest stays on the
// cooperative kernel.
bool rec_f32_supported(int T, int B, int d) {
  return T >= 1 && B >= 1 && d >= 8 && (d & 3) == 0 && d <= RR_WARPS * F32_MAX_KW &&
         (B + F32_NG - 1) / F32_NG <= REC_MAX_DB_ROWS && options().force_generic == 0 && options().rec_reg != 1;
}

int rec_fwd_f32(const RecFwdArgs& a, cudaStream_t stream) {
  RecF32Params p{};
  p.T = a.T; p.B = a.B; p.d = a.d;
  p.W = (const float*)a.W;
  p.in0 = (const float*)a.pre; p.in1 = (const float*)a.g;
  p.self_gate = a.g == nullptr ? 1 : 0;
  p.state = (float*)a.h; p.out0 = (float*)a.v; p.out1 = (float*)a.y;
  return f32_launch(false, p, a.sync, stream);
}

int rec_bwd_f32(const RecBwdArgs& a, cudaStream_t stream) {
  RecF32Params p{};
  p.T = a.T; p.B = a.B; p.d = a.d;
  p.W = (const float*)a.Wt;
  p.self_gate = a.g == nullptr ? 1 : 0;
  p.in0 = (const float*)(a.g != nullptr ? a.g : a.dy); p.in1 = (const float*)a.dy;
  p.in2 = (const float*)a.h; p.in3 = (const float*)a.v;
  p.state = (float*)a.dv; p.out0 = (float*)a.dg; p.db = a.db;
  return f32_launch(true, p, a.sync, stream);
}

}  // namespace elman
