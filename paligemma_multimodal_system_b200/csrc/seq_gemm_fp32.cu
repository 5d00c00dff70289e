// Matrix products of the fp32 serving mode: out[t, f] (+)= (sum_k x[t, k] w[f, k] + bias[f]) * scale, plain fp32 FMAs (no
// reduced-precision tensor mode).
//
// Both operands are K-major, so nothing is transposed: tiles go to shared memory as they lie (cp.async), a thread reads float4s along k
// and every FMA is a packed pair (fma.rn.f32x2) of an even and an odd k.  A sum is therefore two chains of K / 2, added at the
// end -- shorter chains than one in k order, and no closer to bf16 or tf32 anywhere.
//
// (64 x 64 tiles filled by scalar loads without overlap, the form before this one: 3 TFLOP/s over a run of prompts and decode steps.)
//
// Two forms:
//   tile   BM x BN outputs per CTA, a TM x TN register tile per thread, two CTAs of 128 threads per SM (a CTA of 256 with the same thread tile: 44.7
//          TFLOP/s against 47.8; unpacked FMAs 43).  What bounds it is the FMA pipe: a 4-deep k step of the 64 x 128 form is 128 packed FMAs per
//          warp against 16 shared-memory wavefronts.  660 x 2048 . 2048 x 16384: 985 us (45 TFLOP/s).
//   rows   few tokens (decode): the weights are streamed once, straight into registers (a warp owns two or four features, its lanes share
//          out k), the tokens' rows sit in shared memory.  What bounds it is HBM up to four tokens, above that the issue of its FMAs and
//          shared-memory reads.  6 tokens, 16384 x 2048 weights: 27 us (4.9 TB/s).
// Where the output has too few tiles for the SMs, a cluster of up to 8 CTAs shares out k and adds its partial tiles through distributed
// shared memory, rank after rank (the same order in every run).
#include "common.cuh"
#include "paligemma_b200.h"

namespace {

struct Fp32Args {
  const float *x, *w, *bias;
  float* out;
  long long ldx, ldw, ldo, bsx, bsw, bso;
  int T, F, K, kpart;  // kpart: k values per cluster rank (a multiple of the k step)
  int accumulate;
  float scale;
  const int* only_if;  // not NULL: a flag on the device that has to be set for anything to be computed (gemm_fp32_split.cu)
  int early;  // rows kernel: nothing in front writes w (weights_follow), so that its first values may be requested ahead of the dependency wait
};

__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// BYTES (16 or 4) asynchronously from global to shared memory; zeros where `valid` is false (nothing is read)
template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t dst, const float* src, bool valid) {
  const int sz = valid ? BYTES : 0;
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(sz) : "memory");
}

__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float ld_rank(uint32_t addr, uint32_t rank) {  // the same shared-memory offset of CTA `rank` of the cluster
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void finish(const Fp32Args& p, float* out, int t, int f, float v) {
  if (p.bias != nullptr) v += p.bias[f];
  v *= p.scale;
  float* o = out + (long long)t * p.ldo + f;
  if (p.accumulate) v += *o;
  *o = v;
}

constexpr int kStep = 32, kPitch = kStep + 4, kStages = 3;  // a pitch of 36 floats: eight neighbouring rows start in eight different 16-byte banks

// Warps form a WM x WN grid; lane = 4 row positions x 8 column positions, a thread's rows are 4 apart and its columns 8 apart.
template <int WM, int WN, int TM, int TN, int BYTES>
__global__ void __launch_bounds__(WM* WN * 32, 2) gemm_fp32_tile_kernel(Fp32Args p) {
  constexpr int BM = WM * 4 * TM, BN = WN * 8 * TN, NT = WM * WN * 32, EPC = BYTES / 4, CPR = kStep / EPC, RPP = NT / CPR;
  static_assert(BM % RPP == 0 && BN % RPP == 0, "whole passes of the copy over either operand");
  extern __shared__ __align__(16) float sm[];
  const int S = cluster_size(), rank = S > 1 ? pg::cluster_ctarank() : 0;
  const int f0 = (blockIdx.x / S) * BN, t0 = blockIdx.y * BM;
  float* out = p.out + blockIdx.z * p.bso;
  const int k_lo = rank * p.kpart, k_hi = min(p.K, k_lo + p.kpart);
  const int steps = k_hi > k_lo ? (k_hi - k_lo + kStep - 1) / kStep : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ra = (warp / WN) * 4 * TM + (lane >> 3), rb = (warp % WN) * 8 * TN + (lane & 7);
  const uint32_t base = pg::smem_u32(sm);
  // the copy: thread -> one chunk of every RPP-th row
  const int cr = threadIdx.x / CPR, ck = (threadIdx.x % CPR) * EPC;
  const float* xc = p.x + blockIdx.z * p.bsx + (long long)(t0 + cr) * p.ldx + k_lo + ck;
  const float* wc = p.w + blockIdx.z * p.bsw + (long long)(f0 + cr) * p.ldw + k_lo + ck;
  const int xrows = p.T - t0 - cr, wrows = p.F - f0 - cr;
  const uint32_t cdst = base + (cr * kPitch + ck) * 4;
  auto fetch = [&](int step) {
    const uint32_t dst = cdst + (step % kStages) * (BM + BN) * kPitch * 4;
    const bool in = k_lo + step * kStep + ck < k_hi;
#pragma unroll
    for (int r = 0; r < BM; r += RPP) copy_async<BYTES>(dst + r * kPitch * 4, in && r < xrows ? xc + step * kStep + r * p.ldx : p.x, in && r < xrows);
#pragma unroll
    for (int r = 0; r < BN; r += RPP) copy_async<BYTES>(dst + (BM + r) * kPitch * 4, in && r < wrows ? wc + step * kStep + r * p.ldw : p.x, in && r < wrows);
  };
  pg::griddep_wait();
  pg::griddep_launch_dependents();
  if (p.only_if != nullptr && *p.only_if == 0) return;  // (the whole grid)
  float2 acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < steps) fetch(s);
    pg::cp_async_commit();
  }
  for (int s = 0; s < steps; ++s) {
    pg::cp_async_wait<kStages - 2>();
    __syncthreads();  // step s has landed, and every warp is done with the buffer that is refilled now
    if (s + kStages - 1 < steps) fetch(s + kStages - 1);
    pg::cp_async_commit();
    const float* xs = sm + (s % kStages) * (BM + BN) * kPitch + ra * kPitch;
    const float* ws = sm + (s % kStages) * (BM + BN) * kPitch + (BM + rb) * kPitch;
#pragma unroll
    for (int k = 0; k < kStep; k += 4) {
      float4 b[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + 8 * j * kPitch + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(xs + 4 * i * kPitch + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          fma2(acc[i][j], make_float2(a.x, a.y), make_float2(b[j].x, b[j].y));
          fma2(acc[i][j], make_float2(a.z, a.w), make_float2(b[j].z, b[j].w));
        }
      }
    }
  }
  if (S == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (t0 + ra + 4 * i < p.T && f0 + rb + 8 * j < p.F) finish(p, out, t0 + ra + 4 * i, f0 + rb + 8 * j, acc[i][j].x + acc[i][j].y);
    return;
  }
  pg::cp_async_wait<0>();
  __syncthreads();  // the stages become the partial tile [BM][BN]
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sm[(ra + 4 * i) * BN + rb + 8 * j] = acc[i][j].x + acc[i][j].y;
  pg::cluster_sync_all();
  for (int i = rank * NT + threadIdx.x; i < BM * BN; i += S * NT) {
    const int t = t0 + i / BN, f = f0 + i % BN;
    if (t >= p.T || f >= p.F) continue;
    float v = 0.f;
    for (int r = 0; r < S; ++r) v += ld_rank(base + i * 4, r);
    finish(p, out, t, f, v);
  }
  pg::cluster_sync_all();  // nobody leaves while a peer reads its tile
}

// Sums N values per lane over the warp; value i of the result (N <= 32: in lane i * (32 / N); N = 64: values 2 * lane and 2 * lane + 1)
template <int N>
__device__ __forceinline__ void scatter_sum(float (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int n = N;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < N / 2; ++i)
        if (i < n) {
          const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
}

constexpr int kRowsK = 512, kRowsWarps = 8;  // k values of a staged run

// TT token rows, RF features per warp, PF weight steps (RF float4 a lane each) in flight, CTAS per SM
// The first PF steps are under way before the rows are (p.early): with the gate of the feed-forward letting its product come, five requests with 12 decode steps, four
// layers of 2048, 8.79 -> 8.66 ms.
template <int TT, int RF, int PF, int CTAS>
__global__ void __launch_bounds__(kRowsWarps * 32, CTAS) gemm_fp32_rows_kernel(Fp32Args p) {
  extern __shared__ __align__(16) float sm[];  // two runs of TT token rows, [TT][kRowsK]
  const int S = cluster_size(), rank = S > 1 ? pg::cluster_ctarank() : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int f0 = (blockIdx.x / S) * kRowsWarps * RF + warp * RF;
  const float* x = p.x + blockIdx.z * p.bsx;
  const float* w = p.w + blockIdx.z * p.bsw;
  const int k_lo = rank * p.kpart, k_hi = min(p.K, k_lo + p.kpart);
  const int runs = k_hi > k_lo ? (k_hi - k_lo + kRowsK - 1) / kRowsK : 0;
  const uint32_t base = pg::smem_u32(sm);
  auto stage = [&](int run) {
    const uint32_t dst = base + (run & 1) * TT * kRowsK * 4;
    for (int i = threadIdx.x; i < TT * (kRowsK / 4); i += kRowsWarps * 32) {
      const int t = i / (kRowsK / 4), k = k_lo + run * kRowsK + (i % (kRowsK / 4)) * 4;
      const bool valid = t < p.T && k < k_hi;
      copy_async<16>(dst + i * 16, valid ? x + (long long)t * p.ldx + k : p.x, valid);
    }
  };
  const float* wr[RF];
#pragma unroll
  for (int r = 0; r < RF; ++r) wr[r] = w + (long long)min(f0 + r, p.F - 1) * p.ldw;
  auto weights = [&](float4 (&b)[RF], int k) {  // 128 k values of the warp's features; k is the lane's own
#pragma unroll
    for (int r = 0; r < RF; ++r) b[r] = k < k_hi ? __ldcs(reinterpret_cast<const float4*>(wr[r] + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  float2 acc[RF * TT];
#pragma unroll
  for (int i = 0; i < RF * TT; ++i) acc[i] = make_float2(0.f, 0.f);
  float4 b[PF][RF];
  auto request = [&]() {
#pragma unroll
    for (int i = 0; i < PF; ++i) weights(b[i], k_lo + i * 128 + lane * 4);
  };
  if (p.early) request();
  pg::griddep_wait();
  pg::griddep_launch_dependents();
  if (p.only_if != nullptr && *p.only_if == 0) return;  // (the whole grid)
  if (!p.early) request();
  if (runs > 0) stage(0);
  pg::cp_async_commit();
  for (int run = 0; run < runs; ++run) {
    if (run + 1 < runs) stage(run + 1);
    pg::cp_async_commit();
    pg::cp_async_wait<1>();
    __syncthreads();
    const float* xs = sm + (run & 1) * TT * kRowsK + lane * 4;
#pragma unroll
    for (int i = 0; i < kRowsK / 128; ++i) {
      float4 c[RF];
#pragma unroll
      for (int r = 0; r < RF; ++r) c[r] = b[i % PF][r];
      weights(b[i % PF], k_lo + run * kRowsK + (i + PF) * 128 + lane * 4);
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        const float4 a = *reinterpret_cast<const float4*>(xs + t * kRowsK + i * 128);
#pragma unroll
        for (int r = 0; r < RF; ++r) {
          fma2(acc[r * TT + t], make_float2(a.x, a.y), make_float2(c[r].x, c[r].y));
          fma2(acc[r * TT + t], make_float2(a.z, a.w), make_float2(c[r].z, c[r].w));
        }
      }
    }
    __syncthreads();  // the run's buffer is refilled next
  }
  constexpr int N = RF * TT <= 8 ? 8 : RF * TT <= 16 ? 16 : RF * TT <= 32 ? 32 : 64;
  float v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = i < RF * TT ? acc[i].x + acc[i].y : 0.f;
  scatter_sum(v);
  constexpr int PER = N > 32 ? N / 32 : 1, EVERY = N > 32 ? 1 : 32 / N;
  float* out = p.out + blockIdx.z * p.bso;
  if (S == 1) {
    if (lane % EVERY == 0) {
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int i = lane / EVERY * PER + j, t = i % TT, f = f0 + i / TT;
        if (i < RF * TT && t < p.T && f < p.F) finish(p, out, t, f, v[j]);
      }
    }
    return;
  }
  __syncthreads();
  if (lane % EVERY == 0) {
#pragma unroll
    for (int j = 0; j < PER; ++j) sm[warp * N + lane / EVERY * PER + j] = v[j];
  }
  pg::cluster_sync_all();
  for (int i = rank * kRowsWarps * 32 + threadIdx.x; i < kRowsWarps * N; i += S * kRowsWarps * 32) {
    const int t = i % N % TT, f = (blockIdx.x / S) * kRowsWarps * RF + i / N * RF + i % N / TT;
    if (i % N >= RF * TT || t >= p.T || f >= p.F) continue;
    float s = 0.f;
    for (int r = 0; r < S; ++r) s += ld_rank(base + i * 4, r);
    finish(p, out, t, f, s);
  }
  pg::cluster_sync_all();
}

int part(int K, int S, int step) { return ((K + S - 1) / S + step - 1) / step * step; }  // k values of a cluster rank

template <void (*KERNEL)(Fp32Args)>
cudaError_t launch(dim3 grid, int threads, size_t smem, int S, cudaStream_t st, const Fp32Args& p) {
  // (the size belongs to the kernel: set once a device, so that calls of several threads find the same)
  static bool configured[pg::kMaxDevices] = {};
  const int dev = pg::current_device();
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pg_pdl_enabled() ? 2 : 1;
  pg_count_launch(1);
  return cudaLaunchKernelEx(&cfg, KERNEL, p);
}

template <int WM, int WN, int TM, int TN>
cudaError_t launch_tile(bool wide, int S, int batch, cudaStream_t st, const Fp32Args& p) {
  constexpr int BM = WM * 4 * TM, BN = WN * 8 * TN;
  const dim3 grid((p.F + BN - 1) / BN * S, (p.T + BM - 1) / BM, batch);
  if (grid.y > 65535) return cudaErrorInvalidConfiguration;
  const size_t smem = sizeof(float) * kStages * (BM + BN) * kPitch;
  return wide ? launch<gemm_fp32_tile_kernel<WM, WN, TM, TN, 16>>(grid, WM * WN * 32, smem, S, st, p)
              : launch<gemm_fp32_tile_kernel<WM, WN, TM, TN, 4>>(grid, WM * WN * 32, smem, S, st, p);
}

template <int TT, int RF, int PF, int CTAS>
cudaError_t launch_rows(int batch, int sms, cudaStream_t st, Fp32Args p) {
  // clusters share out k until two CTAs per SM are busy or a rank would have less than one staged run
  constexpr int BF = kRowsWarps * RF;
  const int tiles = (p.F + BF - 1) / BF;
  int S = 1;
  while (S < 8 && tiles * batch * S < 2 * sms && p.K >= 2 * S * kRowsK) S *= 2;
  p.kpart = part(p.K, S, kRowsK);
  return launch<gemm_fp32_rows_kernel<TT, RF, PF, CTAS>>(dim3(tiles * S, 1, batch), kRowsWarps * 32, sizeof(float) * 2 * TT * kRowsK, S, st, p);
}

}  // namespace

// The tile and the number of cluster ranks whose busiest SM has the least to do (that in return: outputs times k steps); smaller tiles read shared memory more often per FMA.
static float cheapest_tile(int T, int F, int K, int batch, int& best, int& S) {
  struct Form { int bm, bn; float weight; };
  const Form forms[3] = {{64, 128, 1.0f}, {64, 64, 1.05f}, {32, 64, 1.3f}};
  const int sms = pg::num_sms();
  float least = 0.f;
  best = 0;
  S = 1;
  for (int i = 0; i < 3; ++i) {
    if (i > 0 && (T + forms[i].bm - 1) / forms[i].bm > 65535) break;
    for (int s = 1; s <= 8; s *= 2) {
      if (s > 1 && K < s * 8 * kStep) break;
      const long long ctas = (long long)((F + forms[i].bn - 1) / forms[i].bn) * ((T + forms[i].bm - 1) / forms[i].bm) * batch * s;
      // a rank that joins the others' sums costs about as much as 48 k values more
      const float cost = (float)((ctas + sms - 1) / sms) * forms[i].bm * forms[i].bn * (part(K, s, kStep) + (s > 1 ? 48 : 0)) * forms[i].weight;
      if ((i == 0 && s == 1) || cost < least) { least = cost; best = i; S = s; }
    }
  }
  return least;
}

// us of a product of more than 16 tokens by the tiles (20 tokens to 1000, 64 to 16384 wide and 64 to 8192 deep: half of them within 10 %)
double pg_gemm_fp32_estimate(int T, int F, int K, int accumulate) {
  int best, S;
  return 5.6 + 6.8e-6 * cheapest_tile(T, F, K, 1, best, S) + 0.28e-6 * 4.0 * T * F * (accumulate ? 2 : 1);
}

// batch independent products (bsx / bsw / bso: elements between their operands).  Returns PG_ERR_ARG for what no grid can express.
int pg_gemm_fp32(const float* x, long long ldx, long long bsx, const float* w, long long ldw, long long bsw, float* out, long long ldo, long long bso,
                 const float* bias, int accumulate, float scale, int T, int F, int K, int batch, cudaStream_t st,
                 const int* only_if) {
  Fp32Args p{x, w, bias, out, ldx, ldw, ldo, bsx, bsw, bso, T, F, K, 0, accumulate, scale, only_if, only_if == nullptr ? pg::weights_follow() : 0};
  const int sms = pg::num_sms();
  // 16-byte copies and loads want every row of every operand on a 16-byte boundary
  const bool wide = K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && bsx % 4 == 0 && bsw % 4 == 0 &&
                    ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
  cudaError_t e;
  if (wide && T <= 16) {
    // A warp keeps a pair of sums per feature and token.  Two CTAs of 256 threads on an SM leave a thread 128 registers: four features a warp fit them up to six
    // tokens (48 registers of sums; 32 bytes spill), two features up to eight; nine and more take four features with one CTA per SM.  16384 x 2048 weights: 4
    // tokens 25 us (5.3 TB/s), 6 tokens 27, 8 tokens 36, 16 tokens 51; the 32 x 64 tile takes 66 for 17 .. 32 tokens
    e = T <= 4   ? launch_rows<4, 4, 2, 2>(batch, sms, st, p)
        : T <= 6 ? launch_rows<6, 4, 2, 2>(batch, sms, st, p)
        : T <= 8 ? launch_rows<8, 2, 4, 2>(batch, sms, st, p)
                 : launch_rows<16, 4, 4, 1>(batch, sms, st, p);
  } else {
    int best, S;
    cheapest_tile(T, F, K, batch, best, S);
    p.kpart = part(K, S, kStep);
    e = best == 0   ? launch_tile<2, 2, 8, 8>(wide, S, batch, st, p)
        : best == 1 ? launch_tile<2, 2, 8, 4>(wide, S, batch, st, p)
                    : launch_tile<2, 2, 4, 4>(wide, S, batch, st, p);
  }
  if (e == cudaErrorInvalidConfiguration) return PG_ERR_ARG;
  return e == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}
