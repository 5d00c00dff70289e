// The per-token side input of a decode step in one launch:
//
//   g_j  = gelu_tanh(sum_d G[j, d] a_d) * table[token, col0 + j]     j < n   (rounded to the activation type, as the operand of a product)
//   y_d  = sum_j P[d, j] g_j
//   x   += y / rms(y) * w          (fp32 residual; a, the activation copy of x, follows)
//
// As two products with an element-wise kernel between and a norm behind, a step of 48 rows spent 17 us on it, 0.5 MB of weights: each link is one chain of round
// trips.  Here a cluster of four CTAs has a row: a CTA takes a quarter of the gate outputs, leaves them in its peers' shared memory, takes a quarter of the
// output columns, and the peers exchange one sum of squares.  What bounds it: the four round trips (row, gate weights, peers, projection weights -- requested
// ahead of the exchange), then the weights' way from L2, once per row (so it is for few rows -- token_side_fits in seq_ops.py has the line; beyond, products share
// a weight tile between rows).  Rows of 2048, 64 inner values: 48 bf16 10.7 -> 7.8 us (17 -> 8 in its step), five fp32 9.7 -> 7.3.
#include "common.cuh"
#include "paligemma_b200.h"

using bf16 = __nv_bfloat16;

namespace {

constexpr int kRanks = 4, kThreads = 256, kMaxInner = 256;

__device__ __forceinline__ void get8(const bf16* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void get8(const float* p, float (&v)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ float as_float(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float as_float(float v) { return v; }
__device__ __forceinline__ float rounded(float v, bf16) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float rounded(float v, float) { return v; }
__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void st_peers(float* p, float v) {  // the same word in every CTA of the cluster
  const uint32_t a = pg::smem_u32(p);
#pragma unroll
  for (int r = 0; r < kRanks; ++r) {
    uint32_t d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(r));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(d), "f"(v) : "memory");
  }
}

// act, x, out_act may be one buffer's row (fp32: all three); a row belongs to one cluster, which reads it whole before it writes any of it.
template <typename TA>
__global__ void __launch_bounds__(kThreads) token_side_kernel(const TA* act, const TA* __restrict__ wg, const int* __restrict__ tokens, const TA* __restrict__ table,
                                                              long long ldt, int col0, const TA* __restrict__ wp, const float* __restrict__ norm_w, float* x,
                                                              TA* out_act, int D, int n, int n_pad, float eps, int trigger) {
  extern __shared__ __align__(16) float sm[];
  float* row = sm;           // [D] the activation row
  float* gz = row + D;       // [kMaxInner]
  float* ys = gz + kMaxInner;  // [D / kRanks]
  float* red = ys + D / kRanks;  // [8] warps, [kRanks] ranks
  {  // weights do not depend on the kernels before: on their way to L2 ahead of the wait
    const long long lines = (long long)n_pad * D * sizeof(TA) / 128, i = (long long)blockIdx.x * kThreads + threadIdx.x;
    for (long long l = i; l < lines; l += (long long)gridDim.x * kThreads) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(wg) + l * 128));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(wp) + l * 128));
    }
  }
  pg::griddep_begin_if(trigger);
  const int rank = static_cast<int>(pg::cluster_ctarank()), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long t = blockIdx.x / kRanks;
  const long long tok = tokens[t];
  for (int d = 8 * threadIdx.x; d < D; d += 8 * kThreads) {
    float v[8];
    get8(act + t * D + d, v);
    *reinterpret_cast<float4*>(row + d) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(row + d + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
  __syncwarp();
  pg::cluster_sync_all();  // (the peers are there from here on)
  const int share = (n_pad + kRanks - 1) / kRanks, j1 = min(n_pad, (rank + 1) * share);
  for (int j = rank * share + 2 * warp; j < j1; j += 16) {  // two outputs a warp: their weights are under way together
    const int ja = j, jb = min(j + 1, j1 - 1);
    float a = 0.f, b = 0.f;
#pragma unroll 4
    for (int d = 8 * lane; d < D; d += 256) {
      float u[8], v[8];
      get8(wg + (long long)ja * D + d, u);
      get8(wg + (long long)jb * D + d, v);
      const float4 r0 = *reinterpret_cast<const float4*>(row + d), r1 = *reinterpret_cast<const float4*>(row + d + 4);
      const float r[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) { a = fmaf(u[i], r[i], a); b = fmaf(v[i], r[i], b); }
    }
    a = wsum(a);
    b = wsum(b);
    if (lane < 2 && j + lane < j1) {
      const int jj = j + lane;
      const float z = lane == 0 ? a : b;
      st_peers(gz + jj, jj < n ? rounded(pg::gelu_tanh(z) * as_float(table[tok * ldt + col0 + jj]), TA{}) : 0.f);
    }
  }
  __syncwarp();
  pg::cluster_sync_all();
  // 64 columns a warp: eight lanes share a weight row (eight inner values each), four rows an instruction; the 16 partial sums of a lane are summed by halving
  const int cols = D / kRanks, c0 = rank * cols, kg = lane >> 3, l8 = lane & 7;
  float sq = 0.f;
  for (int cb = 64 * warp; cb < cols; cb += 64 * 8) {
    float s[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = 0.f;
    for (int k = 8 * l8; k < n_pad; k += 64) {
      const float4 g0 = *reinterpret_cast<const float4*>(gz + k), g1 = *reinterpret_cast<const float4*>(gz + k + 4);
      const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float w[8];
        get8(wp + (long long)(c0 + cb + 4 * i + kg) * n_pad + k, w);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[i] = fmaf(w[e], g[e], s[i]);
      }
    }
#pragma unroll
    for (int w = 4, m = 8; w >= 1; w >>= 1, m >>= 1) {
      const bool up = (l8 & w) != 0;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < m) {
          const float mine = up ? s[i + m] : s[i], theirs = up ? s[i] : s[i + m];
          s[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, w);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ys[cb + 4 * (2 * l8 + i) + kg] = s[i];
      sq = fmaf(s[i], s[i], sq);
    }
  }
  sq = wsum(sq);
  if (lane == 0) red[warp] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < 8; ++w) tot += red[w];
    st_peers(red + 8 + rank, tot);
  }
  __syncwarp();
  pg::cluster_sync_all();
  const float inv = 1.0f / sqrtf((red[8] + red[9] + red[10] + red[11]) / (float)D + eps);
  for (int c = 2 * threadIdx.x; c < cols; c += 2 * kThreads) {
    const float2 y = *reinterpret_cast<const float2*>(ys + c), w = *reinterpret_cast<const float2*>(norm_w + c0 + c);
    float2* xp = reinterpret_cast<float2*>(x + t * D + c0 + c);
    float2 v = *xp;
    v.x += y.x * inv * w.x;
    v.y += y.y * inv * w.y;
    *xp = v;
    if (sizeof(TA) == 2 && out_act != nullptr) *reinterpret_cast<uint32_t*>(out_act + t * D + c0 + c) = pg::pack_bf16(v.x, v.y);
  }
}

template <typename TA>
int launch(const void* act, const void* wg, const int* tokens, const void* table, long long ldt, int col0, const void* wp, const float* norm_w, float* x,
           void* out_act, int rows, int D, int n, int n_pad, float eps, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows * kRanks);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (D + kMaxInner + D / kRanks + 8 + kRanks) * sizeof(float);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kRanks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pg_pdl_enabled() ? 2 : 1;
  pg_count_launch(1);
  return cudaLaunchKernelEx(&cfg, token_side_kernel<TA>, static_cast<const TA*>(act), static_cast<const TA*>(wg), tokens, static_cast<const TA*>(table), ldt, col0,
                            static_cast<const TA*>(wp), norm_w, x, static_cast<TA*>(out_act), D, n, n_pad, eps, pg::weights_follow()) == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}

}  // namespace

extern "C" int pg_token_side(const void* act, const void* gate_w, const int* tokens, const void* table, long long ldt, int col0, const void* proj_w,
                             const float* norm_w, float* x, void* out_act, int rows, int D, int n, int n_pad, float eps, int act_f32, void* stream) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(act) | reinterpret_cast<uintptr_t>(gate_w) | reinterpret_cast<uintptr_t>(proj_w) |
                        reinterpret_cast<uintptr_t>(norm_w) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out_act);
  if (act == nullptr || gate_w == nullptr || tokens == nullptr || table == nullptr || proj_w == nullptr || norm_w == nullptr || x == nullptr) return PG_ERR_ARG;
  if (rows <= 0 || rows > 65535 || D <= 0 || D > 8192 || (D % 256) != 0 || n <= 0 || n > n_pad || n_pad > kMaxInner || (n_pad % 8) != 0 || (all & 15) != 0)
    return PG_ERR_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return act_f32 ? launch<float>(act, gate_w, tokens, table, ldt, col0, proj_w, norm_w, x, nullptr, rows, D, n, n_pad, eps, st)
                 : launch<bf16>(act, gate_w, tokens, table, ldt, col0, proj_w, norm_w, x, out_act, rows, D, n, n_pad, eps, st);
}
