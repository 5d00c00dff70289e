// Products of the fp32 serving mode with many tokens, on the tensor cores without giving up fp32: every operand value is cut into three bf16 terms, x = x1 + x2 + x3
// (8 + 8 + 8 significant bits: exact but for values whose last term underflows), and
//
//   x w = x1 w1 + (x1 w2 + x2 w1) + (x2 w2 + x1 w3 + x3 w1)     (what is dropped is below 2^-24 of a product)
//
// runs as six bf16 products.  A tensor core adds into its accumulator with truncation, which over thousands of steps costs more than an fp32 FMA chain; so an accumulator
// holds 64 k values only, smallest terms first, and the epilogue warps add these partial sums in registers, round to nearest, while the next 64 are multiplied.
// Relative error (2-norm) of products of N(0, 1) values against 64 bits, FMAs / here: 2048 deep 2.9e-7 .. 5.7e-7 / 1.1e-7 .. 1.3e-7, 8192 deep 4.1e-7 / 1.5e-7.
//
// Three launches: split (both operands into planes of a scratch the caller owns), product, and -- where the output has too few tiles for the SMs, K is shared out
// between pairs of CTAs -- a sum of the partial outputs, part after part.  Infinities and NaNs have no such split, and where products come near the end of the range one
// term may overflow to either side and the sum of two be no number (inf - inf).  So the split kernel raises a flag for values so large that a
// sum could reach 2^127 (safe_exponent; 2^57 for K = 2048), the product then writes nothing, and the plain-FMA kernel launched behind it, which otherwise returns at once,
// computes the call.  (A bound of the operands' largest exponents together would let more through; their maxima as atomics cost a decode burst of five requests 8 %.)
//
// What it holds: operands above about 1e-33 keep their 24 bits; below, the third term and then the second fall under the smallest bf16 (at 2e-36 16 bits are left).
//
// CTA pair per 256 x 256 tile (cta_group::2) as in gemm_tcgen05.cu; a stage is three planes of 128 token rows and three of 128 feature rows, 96 KB for
// 24 UMMAs of 256 x 256 x 16 (1536 clocks), so what an SM takes in (62 bytes a clock) and the tensor pipe are balanced.  What bounds it: both.
// us, FMAs / here: 750 tokens 16384 x 2048 1100 / 304, 2048 x 8192 627 / 156, 2048 x 2048 170 / 56; 256 tokens 8192 x 2048 222 / 90; 128 tokens 2048 x 8192 120 / 83.
// Five requests in fp32, prompts of 150 tokens and 12 steps: 15.8 -> 8.8 ms, and half the error against 64 bits (6e-7 -> 3e-7).
#include "common.cuh"
#include "paligemma_b200.h"
#include "tmap.cuh"

// seq_gemm_fp32.cu; only_if: the call is computed only where this flag is set
int pg_gemm_fp32(const float* x, long long ldx, long long bsx, const float* w, long long ldw, long long bsw, float* out, long long ldo, long long bso,
                 const float* bias, int accumulate, float scale, int T, int F, int K, int batch, cudaStream_t st, const int* only_if);
double pg_gemm_fp32_estimate(int T, int F, int K, int accumulate);  // us of the plain-FMA form

namespace pg {
namespace {

constexpr int kRows = 128, kTile = 256, kKb = 64, kPlane = kRows * kKb * 2, kOperand = 3 * kPlane, kStage = 2 * kOperand, kStages = 2, kThreads = 320;
constexpr int kSmem = kStages * kStage + 256;

// one value as three bf16: nearest first (truncated where that would be infinite), the remainders exact
PG_DEVINL void split3(float v, uint32_t& a, uint32_t& b, uint32_t& c) {
  const uint32_t u = __float_as_uint(v);
  const uint32_t r = (u & 0x7fffffffu) >= 0x7f7f0000u ? u : u + 0x7fffu + ((u >> 16) & 1);
  a = r >> 16;
  const float v2 = v - __uint_as_float(r & 0xffff0000u);
  const uint32_t u2 = __float_as_uint(v2), r2 = u2 + 0x7fffu + ((u2 >> 16) & 1);
  b = r2 >> 16;
  const float v3 = v2 - __uint_as_float(r2 & 0xffff0000u);
  const uint32_t u3 = __float_as_uint(v3);
  c = (u3 + 0x7fffu + ((u3 >> 16) & 1)) >> 16;
}

// The largest biased exponent of an operand that cannot bring a sum to 2^127: a value is below 2^(e - 126), the six terms of a product are together below 1.02 times that of
// their operands, and K of them are added, so 2 e + log2 K is at most 378.
int safe_exponent(int K) {
  int log_k = 0;
  while (log_k < 31 && (1LL << log_k) < K) ++log_k;
  return (378 - log_k) / 2;
}

// rows of x, then rows of w -> planes [3][T][K] and [3][F][K]; eight values a thread
__global__ void __launch_bounds__(256) fp32_split_kernel(const float* __restrict__ x, long long ldx, int T, const float* __restrict__ w, long long ldw, int F, int K,
                                                         uint4* __restrict__ xp, uint4* __restrict__ wp, int* __restrict__ flag, int safe) {
  griddep_wait();
  const int per = K / 8;
  const long long id = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x, nx = static_cast<long long>(T) * per, nw = static_cast<long long>(F) * per;
  if (id >= nx + nw) return;
  const bool is_x = id < nx;
  const long long i = is_x ? id : id - nx, n = is_x ? nx : nw;
  const float* src = (is_x ? x + i / per * ldx : w + i / per * ldw) + i % per * 8;
  const float4 p = reinterpret_cast<const float4*>(src)[0], q = reinterpret_cast<const float4*>(src)[1];
  const float v[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
  uint32_t o[3][8];
  bool large = false;  // (infinities and NaNs have the largest exponent)
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    large = large || static_cast<int>((__float_as_uint(v[k]) & 0x7f800000u) >> 23) > safe;
    split3(v[k], o[0][k], o[1][k], o[2][k]);
  }
  uint4* dst = (is_x ? xp : wp) + i;
#pragma unroll
  for (int t = 0; t < 3; ++t)
    dst[t * n] = make_uint4(o[t][0] | o[t][1] << 16, o[t][2] | o[t][3] << 16, o[t][4] | o[t][5] << 16, o[t][6] | o[t][7] << 16);
  if (large) *flag = 1;
}

struct SplitArgs {
  float* out;        // split_k 1: the output, else the partial outputs [split_k][T][F]
  const float* bias;
  const int* flag;
  long long ldo;
  int T, F, K, split_k, accumulate;
  float scale;
};

PG_DEVINL float4 finished(float4 v, const float* bias, float scale, const float* old) {
  if (bias != nullptr) { v.x += bias[0]; v.y += bias[1]; v.z += bias[2]; v.w += bias[3]; }
  v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
  if (old != nullptr) { v.x += old[0]; v.y += old[1]; v.z += old[2]; v.w += old[3]; }
  return v;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
fp32_split_gemm_kernel(const __grid_constant__ CUtensorMap tmapX, const __grid_constant__ CUtensorMap tmapW, const SplitArgs args) {
  constexpr uint32_t IDESC = make_idesc_bf16(kTile, kTile);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  if ((smem_base & 1023u) != 0) __trap();
  const uint32_t bar_base = smem_base + kStages * kStage;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
  auto tfull_bar = [&](int s) { return bar_base + 8u * (2 * kStages + s); };
  auto tempty_bar = [&](int s) { return bar_base + 8u * (2 * kStages + 2 + s); };
  const uint32_t tmem_slot = bar_base + 8u * (2 * kStages + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = static_cast<int>(cluster_ctarank());
  const bool leader = rank == 0;
  const int m_blocks = (args.T + kTile - 1) / kTile, n_blocks = (args.F + kTile - 1) / kTile, total_kb = (args.K + kKb - 1) / kKb;
  const int per = (total_kb + args.split_k - 1) / args.split_k, num_tiles = m_blocks * n_blocks * args.split_k;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  // token blocks of one feature block side by side: its weights are read from memory once
  auto tile_at = [&](int tile, int& m, int& n, int& part) {
    m = tile % m_blocks;
    n = tile / m_blocks % n_blocks;
    part = tile / (m_blocks * n_blocks);
  };

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmapX);
    tma_prefetch_desc(&tmapW);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tfull_bar(s), 1);
      mbar_init(tempty_bar(s), 16);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot) : "memory");
  griddep_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = pair; tile < num_tiles; tile += pairs) {
        int m, n, part;
        tile_at(tile, m, n, part);
        const int kb1 = min(total_kb, (part + 1) * per);
        for (int kb = part * per; kb < kb1; ++kb) {
          const uint32_t sa = smem_base + stage * kStage;
          mbar_wait(empty_bar(stage), phase ^ 1);
          if (leader) mbar_expect_tx(full_bar(stage), 2 * kStage);
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            tma_load_2d_pair(sa + p * kPlane, &tmapX, full_bar(stage), kb * kKb, p * args.T + (2 * m + rank) * kRows, kEvictNormal);
            tma_load_2d_pair(sa + kOperand + p * kPlane, &tmapW, full_bar(stage), kb * kKb, p * args.F + (2 * n + rank) * kRows, kEvictNormal);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (leader) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int tile = pair; tile < num_tiles; tile += pairs) {
        int m, n, part;
        tile_at(tile, m, n, part);
        const int kb1 = min(total_kb, (part + 1) * per);
        for (int kb = part * per; kb < kb1; ++kb) {
          mbar_wait(tempty_bar(acc), acc_phase ^ 1);
          mbar_wait(full_bar(stage), phase);
          tc_fence_after();
          const uint32_t sa = smem_base + stage * kStage, d = tmem_base + acc * kTile;
          if (elect_one()) {
            constexpr int PX[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};  // the smallest terms first
#pragma unroll
            for (int t = 0; t < 6; ++t) {
              const uint64_t xd = make_sdesc_k_sw128(sa + PX[t] * kPlane), wd = make_sdesc_k_sw128(sa + kOperand + PW[t] * kPlane);
#pragma unroll
              for (int k = 0; k < kKb / 16; ++k) umma_f16_pair(d, xd + 2 * k, wd + 2 * k, IDESC, (t > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit_pair(empty_bar(stage));
            umma_commit_pair(tfull_bar(acc));
          }
          __syncwarp();
          if (++stage == kStages) { stage = 0; phase ^= 1; }
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * 128;
    const bool write = *args.flag == 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < num_tiles; tile += pairs) {
      int m, n, part;
      tile_at(tile, m, n, part);
      const int kb0 = part * per, kb1 = min(total_kb, kb0 + per);
      float sum[128];
#pragma unroll
      for (int i = 0; i < 128; ++i) sum[i] = 0.f;
#pragma unroll 1
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(tfull_bar(acc), acc_phase);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 128; c += 16) {
          uint32_t r[16];
          tmem_ld16(lanes + acc * kTile + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) sum[c + i] += __uint_as_float(r[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(tempty_bar(acc));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      const int t = (2 * m + rank) * kRows + q * 32 + lane, f0 = n * kTile + half * 128;
      if (write && t < args.T) {
        const bool whole = args.split_k == 1;
        float* o = args.out + (whole ? t * args.ldo : (static_cast<long long>(part) * args.T + t) * args.F) + f0;
#pragma unroll
        for (int i = 0; i < 128; i += 4) {
          if (f0 + i >= args.F) continue;  // (host: F % 4 == 0)
          float4 v = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
          if (whole) v = finished(v, args.bias == nullptr ? nullptr : args.bias + f0 + i, args.scale, args.accumulate ? o + i : nullptr);
          *reinterpret_cast<float4*>(o + i) = v;
        }
      }
    }
  }
  tc_fence_before();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

__global__ void __launch_bounds__(256) fp32_split_sum_kernel(const float* __restrict__ part, SplitArgs args, float* __restrict__ out) {
  griddep_wait();
  if (*args.flag != 0) return;
  const long long id = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x, n = static_cast<long long>(args.T) * args.F;
  if (4 * id >= n) return;
  const long long t = 4 * id / args.F;
  const int f = static_cast<int>(4 * id % args.F);
  float4 v = *reinterpret_cast<const float4*>(part + 4 * id);
  for (int s = 1; s < args.split_k; ++s) {
    const float4 u = *reinterpret_cast<const float4*>(part + s * n + 4 * id);
    v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
  }
  float* o = out + t * args.ldo + f;
  *reinterpret_cast<float4*>(o) = finished(v, args.bias == nullptr ? nullptr : args.bias + f, args.scale, args.accumulate ? o : nullptr);
}

// How a call is cut, and whether it is the faster form.  The split of the weights (10 bytes a value) is what few tokens pay for, the rows what a short K pays for.  Both sides
// are estimated in us; the constants were fitted to 1836 products timed in turn on both sides (32 .. 1000 tokens, 64 .. 16384 x 64 .. 8192), with this line 1.0 % slower on
// average than the better side each time.  us, FMAs / here: 64 tokens 16384 x 2048 116 / 141, 128 tokens 8192 x 2048 115 / 85; 200 tokens 1024 x 1024 25 / 26,
// 512 x 8192 109 / 48; added to an output: 750 tokens 16384 x 64 74 / 100, 400 tokens 2048 x 512 31 / 58.
struct Plan { int split_k; bool use; };
Plan plan(int T, int F, int K, int accumulate) {
  const int pairs = num_sms() / 2, kb = (K + kKb - 1) / kKb, tiles = ((T + kTile - 1) / kTile) * ((F + kTile - 1) / kTile);
  Plan best{1, false};
  double least = 0;
  int steps = 0;  // 64-deep steps of the busiest pair
  for (int s = 1; s <= 16 && s <= kb; ++s) {
    const int per = (kb + s - 1) / s;
    if ((kb + per - 1) / per != s) continue;  // no empty part
    const int rounds = (tiles * s + pairs - 1) / pairs;
    const double clocks = rounds * (per * 1700.0 + 6000.0) + (s > 1 ? 4000.0 + 4.0 * (s + 1) * T * F / 2500.0 : 0.0);
    if (s == 1 || clocks < least) { least = clocks; best.split_k = s; steps = rounds * per; }
  }
  const double mb = 4e-6 * T * F;
  const double ours = 18.7 + 1.95e-6 * (static_cast<double>(F) + T) * K + 2.0 * steps + 0.67 * mb * (accumulate ? 2 : 1) + (best.split_k > 1 ? 0.16 * mb * (best.split_k + 1) : 0.0);
  best.use = ours < 0.9 * pg_gemm_fp32_estimate(T, F, K, accumulate);
  return best;
}

long long scratch_of(int T, int F, int K, int split_k) { return 16 + 6LL * (static_cast<long long>(T) + F) * K + (split_k > 1 ? 4LL * split_k * T * F : 0); }

// The planes are half as large again as the operands.  A call takes at most 256 MB of scratch, whatever its operands: larger ones (a vocabulary) go in blocks of whole
// tiles that use it one after the other.  Where not even one tile fits the plain FMAs compute the call.  (750 tokens x 16384 x 2048 takes 211 MB.)
constexpr long long kMaxScratch = 256LL << 20;

struct Blocks { int tokens, features; Plan plan; };  // of one block; tokens 0: none fits
Blocks blocks(int T, int F, int K, int accumulate) {
  Blocks b{T, F, plan(T, F, K, accumulate)};
  while (scratch_of(b.tokens, b.features, K, b.plan.split_k) > kMaxScratch) {
    int& larger = b.tokens > b.features ? b.tokens : b.features;
    if (larger <= kTile) return Blocks{0, 0, Plan{1, false}};
    larger = ((larger + 1) / 2 + kTile - 1) / kTile * kTile;
    b.plan = plan(b.tokens, b.features, K, accumulate);
  }
  return b;
}

}  // namespace
}  // namespace pg

static long long scratch_where_faster(int tokens, int features, int K, int accumulate) {
  if (tokens < 32 || features < 64 || K < 64 || K % 8 != 0 || features % 4 != 0) return 0;
  const pg::Blocks b = pg::blocks(tokens, features, K, accumulate);
  return b.plan.use ? pg::scratch_of(b.tokens, b.features, K, b.plan.split_k) : 0;
}
extern "C" long long pg_gemm_fp32_scratch(int tokens, int features, int K) { return scratch_where_faster(tokens, features, K, 0); }
extern "C" long long pg_gemm_fp32_scratch_add(int tokens, int features, int K) { return scratch_where_faster(tokens, features, K, 1); }

namespace pg {
namespace {
// one block of the call
int split_block(const float* x, long long ldx, const float* w, long long ldw, float* out, long long ldo, const float* bias, int accumulate, float scale, int tokens, int features,
                int K, void* scratch, long long scratch_bytes, cudaStream_t st) {
  int split_k = plan(tokens, features, K, accumulate).split_k;
  if (scratch_bytes < scratch_of(tokens, features, K, split_k)) split_k = 1;  // (the last block of a row: its parts may want more than a whole block does)
  const long long xn = 3LL * tokens * K * 2, wn = 3LL * features * K * 2;
  char* s = static_cast<char*>(scratch);
  int* flag = reinterpret_cast<int*>(s);
  uint4* xp = reinterpret_cast<uint4*>(s + 16);
  uint4* wp = reinterpret_cast<uint4*>(s + 16 + xn);
  float* part = reinterpret_cast<float*>(s + 16 + xn + wn);
  static bool configured[kMaxDevices] = {};
  const int dev = current_device();
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(fp32_split_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) {
      cudaGetLastError();
      return PG_ERR_CUDA;
    }
    configured[dev] = true;
  }
  CUtensorMap tx, tw;
  int rc;
  if ((rc = make_tmap_2d(&tx, xp, 3LL * tokens, K, K, kRows)) != PG_OK) return rc;
  if ((rc = make_tmap_2d(&tw, wp, 3LL * features, K, K, kRows)) != PG_OK) return rc;
  if (cudaMemsetAsync(flag, 0, sizeof(int), st) != cudaSuccess) {
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  const long long pieces = (static_cast<long long>(tokens) + features) * (K / 8);
  if (launch_kernel(fp32_split_kernel, dim3(static_cast<unsigned>((pieces + 255) / 256)), dim3(256), 0, st, x, ldx, tokens, w, ldw, features, K, xp, wp, flag, safe_exponent(K)) != cudaSuccess)
    return PG_ERR_CUDA;
  SplitArgs a{split_k > 1 ? part : out, bias, flag, ldo, tokens, features, K, split_k, accumulate, scale};
  const int tiles = ((tokens + kTile - 1) / kTile) * ((features + kTile - 1) / kTile) * split_k, pairs = num_sms() / 2;
  if (launch_kernel(fp32_split_gemm_kernel, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(kThreads), kSmem, st, tx, tw, a) != cudaSuccess) return PG_ERR_CUDA;
  if (split_k > 1 &&
      launch_kernel(fp32_split_sum_kernel, dim3(static_cast<unsigned>((static_cast<long long>(tokens) * features / 4 + 255) / 256)), dim3(256), 0, st, part, a, out) != cudaSuccess)
    return PG_ERR_CUDA;
  return pg_gemm_fp32(x, ldx, 0, w, ldw, 0, out, ldo, 0, bias, accumulate, scale, tokens, features, K, 1, st, flag);
}
}  // namespace
}  // namespace pg

extern "C" int pg_gemm_fp32_split(const float* x, long long ldx, const float* w, long long ldw, float* out, long long ldo, const float* bias, int accumulate, float scale,
                                  int tokens, int features, int K, void* scratch, long long scratch_bytes, void* stream) {
  using namespace pg;
  if (tokens <= 0 || features <= 0 || K <= 0 || x == nullptr || w == nullptr || out == nullptr || scratch == nullptr) return PG_ERR_ARG;
  const uintptr_t all = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(scratch);
  if (K % 8 != 0 || features % 4 != 0 || ldx % 4 != 0 || ldw % 4 != 0 || ldo % 4 != 0 || (all & 15) != 0) return PG_ERR_ARG;
  const Blocks b = blocks(tokens, features, K, accumulate);
  if (b.tokens == 0 || scratch_bytes < scratch_of(b.tokens, b.features, K, b.plan.split_k)) return PG_ERR_ARG;
  for (long long t = 0; t < tokens; t += b.tokens)
    for (long long f = 0; f < features; f += b.features) {
      const int nt = static_cast<int>(tokens - t < b.tokens ? tokens - t : b.tokens), nf = static_cast<int>(features - f < b.features ? features - f : b.features);
      const int rc = split_block(x + t * ldx, ldx, w + f * ldw, ldw, out + t * ldo + f, ldo, bias == nullptr ? nullptr : bias + f, accumulate, scale, nt, nf, K, scratch,
                                 scratch_bytes, reinterpret_cast<cudaStream_t>(stream));
      if (rc != PG_OK) return rc;
    }
  return PG_OK;
}
