// Single-precision GEMM with arbitrary element strides on the CUDA cores:
//   C[m,n] = sum_k A(m,k) B(k,n) (+ bias[n]) (+ C[m,n])
// fp32 products and sums: the parity path of the library (the reference calls cuBLAS,
// elman/cuda/lib/blas.h:25-50).
//
// 64 x 64 tiles, 4 x 4 outputs per thread, K in slabs of 16 through two shared-memory buffers: the
// next slab is on its way into registers while the current one is multiplied.  The fp32 products of
// this path are small (a few hundred rows and columns), so their tiles alone leave most of the
// device idle and each would walk the whole K behind its own load latency: a thread-block cluster
// of S CTAs shares a tile, each takes a contiguous part of K, and the partial tiles meet over
// distributed shared memory in rank order (deterministic, no scratch in memory).  S is the
// largest of 1, 2, 4, 8 that keeps the grid within four CTAs per SM and 64 columns of K per CTA.
//
// Measured (us, one-tile kernel before -> now):
//   512 x 256 x 256        43 -> 7.0
//   256 x 256 x 512 (TN)  ~85 -> 7.6
//   1600 x 512 x 512       96 -> 33
#include "common.cuh"

namespace elman {

namespace {

constexpr int FT = 64, FK = 16, FPAD = FT + 4, FMAX_S = 8;

// One thread's float4 of a [64 x 16] operand slab.  UNIT_K: consecutive elements run along K.
template <bool UNIT_K, bool VEC>
__device__ __forceinline__ float4 slab_load(const float* __restrict__ P, long s_row, long s_k, int r0,
                                            int rows, int k0, int k_end, int tid) {
  const int r = r0 + (UNIT_K ? tid >> 2 : (tid & 15) * 4);
  const int k = k0 + (UNIT_K ? (tid & 3) * 4 : tid >> 4);
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (UNIT_K) {
    if (r >= rows) return v;
    const float* p = P + r * s_row + k;
    if (VEC && k + 4 <= k_end) return __ldg(reinterpret_cast<const float4*>(p));
    if (k < k_end) v.x = __ldg(p);
    if (k + 1 < k_end) v.y = __ldg(p + 1);
    if (k + 2 < k_end) v.z = __ldg(p + 2);
    if (k + 3 < k_end) v.w = __ldg(p + 3);
  } else {
    if (k >= k_end) return v;
    const float* p = P + k * s_k + r * s_row;     // s_row is 1 unless neither stride is
    if (VEC && r + 4 <= rows) return __ldg(reinterpret_cast<const float4*>(p));
    if (r < rows) v.x = __ldg(p);
    if (r + 1 < rows) v.y = __ldg(p + s_row);
    if (r + 2 < rows) v.z = __ldg(p + 2 * s_row);
    if (r + 3 < rows) v.w = __ldg(p + 3 * s_row);
  }
  return v;
}
template <bool UNIT_K>
__device__ __forceinline__ void slab_store(float (*S)[FPAD], const float4& v, int tid) {
  if (UNIT_K) {
    const int r = tid >> 2, k = (tid & 3) * 4;
    S[k][r] = v.x; S[k + 1][r] = v.y; S[k + 2][r] = v.z; S[k + 3][r] = v.w;
  } else {
    *reinterpret_cast<float4*>(&S[tid >> 4][(tid & 15) * 4]) = v;
  }
}

template <bool AK, bool BK, bool VEC>
__global__ void __launch_bounds__(256)
gemm_f32_kernel(int M, int N, int K, int k_per, const float* __restrict__ A, long sAm, long sAk,
                const float* __restrict__ B, long sBk, long sBn, const float* __restrict__ bias,
                float* __restrict__ C, long ldc, int accumulate) {
  __shared__ __align__(16) float sm[2][2][FK][FPAD];     // [buffer][operand]; then the partial tile
  float* tile = &sm[0][0][0][0];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.z * FT, n0 = blockIdx.y * FT;
  const int S = gridDim.x, rank = blockIdx.x;             // the cluster is the x dimension
  const int kb = rank * k_per, ke = kb + k_per < K ? kb + k_per : K;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  if (kb < ke) {
    float4 a = slab_load<AK, VEC>(A, sAm, sAk, m0, M, kb, ke, tid);
    float4 b = slab_load<BK, VEC>(B, sBn, sBk, n0, N, kb, ke, tid);
    int buf = 0;
    for (int k0 = kb; k0 < ke; k0 += FK, buf ^= 1) {
      slab_store<AK>(sm[buf][0], a, tid);
      slab_store<BK>(sm[buf][1], b, tid);
      __syncthreads();      // two buffers: the next slab's stores wait for nobody's reads of this one
      if (k0 + FK < ke) {
        a = slab_load<AK, VEC>(A, sAm, sAk, m0, M, k0 + FK, ke, tid);
        b = slab_load<BK, VEC>(B, sBn, sBk, n0, N, k0 + FK, ke, tid);
      }
#pragma unroll
      for (int k = 0; k < FK; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(&sm[buf][0][k][ty * 4]);
        const float4 y = *reinterpret_cast<const float4*>(&sm[buf][1][k][tx * 4]);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xs[i], ys[j], acc[i][j]);
      }
    }
  }
  auto put = [&](int gm, int gn, float v) {
    if (bias != nullptr) v += __ldg(bias + gn);
    float* c = C + gm * ldc + gn;
    *c = accumulate ? *c + v : v;
  };
  if (S == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int gm = m0 + ty * 4 + i, gn = n0 + tx * 4 + j;
        if (gm < M && gn < N) put(gm, gn, acc[i][j]);
      }
    return;
  }
  // ---- partial tiles meet: CTA `rank` finishes 64 / S rows ----
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(tile + (ty * 4 + i) * FT + tx * 4) =
        make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int rows = FT / S, base = rank * rows;
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(tile);
  for (int e = tid; e < rows * FT; e += 256) {
    const int m = base + e / FT, n = e % FT;
    if (m0 + m >= M || n0 + n >= N) continue;
    float v = 0.f;
    for (int r = 0; r < S; ++r) {
      uint32_t at;
      float x;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine + (m * FT + n) * 4), "r"(r));
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at));
      v += x;
    }
    put(m0 + m, n0 + n, v);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace

int gemm_f32(int M, int N, int K, const float* A, long sAm, long sAk, const float* B, long sBk, long sBn,
             const float* bias, float* C, long ldc, int accumulate, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return ELMAN_OK;
  const int gm = (M + FT - 1) / FT, gn = (N + FT - 1) / FT;
  if (gm > 65535 || gn > 65535) return ELMAN_ERR_UNSUPPORTED;
  const bool ak = sAk == 1, bk = sBk == 1;
  if ((!ak && sAm != 1) || (!bk && sBn != 1)) return ELMAN_ERR_UNSUPPORTED;
  const bool vec = (((uintptr_t)A | (uintptr_t)B) & 15) == 0 && ((ak ? sAm : sAk) & 3) == 0 &&
                   ((bk ? sBn : sBk) & 3) == 0;
  int S = 1;
  while (S < FMAX_S && (long)gm * gn * S * 2 <= 4L * rec_reg_sms() && K >= 64 * 2 * S) S *= 2;
  int k_per = (K + S - 1) / S;
  k_per = (k_per + FK - 1) / FK * FK;
  void (*kern)(int, int, int, int, const float*, long, long, const float*, long, long, const float*,
               float*, long, int) = nullptr;
  if (ak && bk) kern = vec ? gemm_f32_kernel<true, true, true> : gemm_f32_kernel<true, true, false>;
  else if (ak) kern = vec ? gemm_f32_kernel<true, false, true> : gemm_f32_kernel<true, false, false>;
  else if (bk) kern = vec ? gemm_f32_kernel<false, true, true> : gemm_f32_kernel<false, true, false>;
  else kern = vec ? gemm_f32_kernel<false, false, true> : gemm_f32_kernel<false, false, false>;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(S, gn, gm);
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = S;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = S > 1 ? 1 : 0;
  ELMAN_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, M, N, K, k_per, A, sAm, sAk, B, sBk, sBn, bias, C, ldc,
                                      accumulate));
  count_launch(false);
  return ELMAN_OK;
}

}  // namespace elman
