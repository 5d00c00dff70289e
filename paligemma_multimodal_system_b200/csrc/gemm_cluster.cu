// Products of a moderate number of tokens, below what fills the GPU with 256-wide token tiles: one image, one prompt, one mixed step of the serving engine (up to
// 1408 tokens, with K <= 128 up to 4096), and decode steps of up to 128 tokens whose grid is one wave.  cluster_form in gemm_tcgen05.cu gives the lines and
// both sides of them.  In its grouped form the same kernel walks the routing plan of the experts.
//
//   out[t, f] = epilogue(sum_k X[t, k] W[f, k])       X [tokens, K], W [features, K] bf16, fp32 accumulation
//
// What bounds such a product is the chain of one tile (dependency wait, first bytes, K / 64 pipeline steps, epilogue) and, for long weights, the
// 64 bytes a clock that an SM takes in from L2 -- not the tensor pipe.  So:
//   * weights sit on the UMMA M axis (128 features), a tile's tokens on N, up to 384 in steps of 16: no padding to 128-token rows, and every
//     weight tile is read once per token tile, where 128-row token tiles read it two or three times;
//   * a cluster of up to 8 CTAs shares out K of one tile.  The partial tiles meet in shared memory: every rank adds up a share of the tokens
//     through distributed shared memory, rank after rank (the same sum in every run, no atomics, no zeroed accumulator), and
//     finishes that share, so the epilogue is spread over the cluster, too;
//   * the exchange tile is [token][128 features], written from tensor memory without bank conflicts and read in whole rows, so outputs, residual
//     rows and gate / up pairs are moved as full lines by all eight epilogue warps.
// One tile per CTA; warp 1 = tcgen05.mma issuer + TMEM owner, warps 2..9 = epilogue, warp 0 and, until the tile is summed, the first of those = TMA producers: one issuing thread turns a
// stage around in about 290 ns whatever lies in it, and kProducers of them side by side as many stages: 263 x 2048 x 16384 28.1 -> 26.5 us, 48 x 16384 x 2048 14.7 -> 14.2,
// 706 x 2048 x 2048 13.9 -> 13.2, four encoder layers of one image 229 -> 218.  (A stage keeps its producer, which has seen every phase of the barrier that it waits on.)
#include "common.cuh"
#include "gemm_act.cuh"
#include "gemm_cluster.h"
#include "paligemma_b200.h"
#include "tmap.cuh"

namespace pg {
namespace {

constexpr int kFeat = 128, kKb = 64, kATile = kFeat * kKb * 2, kThreads = 320, kMaxSplit = 8;
constexpr int kProducers = 4;  // warp 0 and warps 2 .. kProducers: every kProducers-th stage each
constexpr int kSmemMax = 232448 - 256;  // barriers behind the stages

PG_DEVINL float4 ld_cluster4(uint32_t addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// sum over the ranks, in their order, of four neighbouring features of one token (all reads under way together)
template <bool SPLIT>
PG_DEVINL float4 gather4(uint32_t addr, int S) {
  if (!SPLIT) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
  }
  float4 u[kMaxSplit];
#pragma unroll
  for (int r = 0; r < kMaxSplit; ++r)
    if (r < S) u[r] = ld_cluster4(addr, r);
  float4 v = u[0];
#pragma unroll
  for (int r = 1; r < kMaxSplit; ++r)
    if (r < S) { v.x += u[r].x; v.y += u[r].y; v.z += u[r].z; v.w += u[r].w; }
  return v;
}

// GROUPED: a CTA takes a tile of a device-side plan (one expert's rows); everything it reads may come from the kernel before, the plan included.
template <bool SPLIT, bool GROUPED = false>
__global__ void __launch_bounds__(kThreads, GROUPED ? 2 : 1) gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmapW, const __grid_constant__ CUtensorMap tmapX,
                                                                   const ClusterGemmArgs args) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  if ((smem_base & 1023u) != 0) __trap();
  constexpr int kU = SPLIT ? 2 : 4;  // tokens a thread finishes together
  const int S = SPLIT ? args.split : 1, rank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
  const int f0 = (blockIdx.x / S) * kFeat;
  int t0 = blockIdx.y * args.tile_tokens, w0 = f0, t_end = args.tokens;  // first token and weight row of the tile, end of its tokens
  if (GROUPED) {
    griddep_wait();
    if (static_cast<int>(blockIdx.y) >= args.plan[0]) return;
    const int* tile = args.plan + 4 + 3 * blockIdx.y;
    w0 += tile[0] * args.features;
    t0 = tile[1];
    t_end = t0 + tile[2];
  }
  const int stages = args.stages, stage_bytes = kATile + args.tile_tokens * 128;
  const int total_kb = (args.K + kKb - 1) / kKb, per = (total_kb + S - 1) / S;
  const int kb0 = rank * per, nkb = min(total_kb, kb0 + per) - kb0;  // (host: no empty rank)
  const uint32_t bar_base = smem_base + args.smem_tiles;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (8 + s); };
  const uint32_t done_bar = bar_base + 8u * 16, tmem_slot = bar_base + 8u * 17;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = args.tile_tokens > 256 ? args.tile_tokens / 2 : args.tile_tokens, chunks = args.tile_tokens > 256 ? 2 : 1;
  const uint32_t cols = args.tile_tokens <= 32 ? 32 : args.tile_tokens <= 64 ? 64 : args.tile_tokens <= 128 ? 128 : args.tile_tokens <= 256 ? 256 : 512;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmapW);
    tma_prefetch_desc(&tmapX);
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot) : "memory");

  auto produce = [&](int first) {
    if (lane == 0) {
      const int pre = min(stages, nkb);
      for (int kb = first; kb < pre; kb += kProducers) {  // weights do not depend on the kernel before: requested ahead of the dependency wait
        mbar_expect_tx(full_bar(kb), stage_bytes);
        tma_load_2d(smem_base + kb * stage_bytes, &tmapW, full_bar(kb), (kb0 + kb) * kKb, w0, kEvictNormal);
      }
      if (!GROUPED) griddep_wait();
      if (first == 0) griddep_launch_dependents();
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < nkb; ++kb, stage = stage + 1 == stages ? 0 : stage + 1, phase ^= stage == 0 ? 1u : 0u) {
        if (stage % kProducers != first) continue;  // a stage has one producer: it has seen every earlier phase of the barrier that it waits on
        const uint32_t sa = smem_base + stage * stage_bytes;
        if (kb >= pre) {
          mbar_wait(empty_bar(stage), phase ^ 1);
          mbar_expect_tx(full_bar(stage), stage_bytes);
          tma_load_2d(sa, &tmapW, full_bar(stage), (kb0 + kb) * kKb, w0, kEvictNormal);
        }
        for (int c = 0; c < chunks; ++c)
          tma_load_2d(sa + kATile + c * chunk * 128, &tmapX, full_bar(stage), (kb0 + kb) * kKb, t0 + c * chunk, kEvictLast);
      }
    }
    __syncwarp();
  };
  if (warp == 0) {
    produce(0);
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc_bf16(kFeat, chunk);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < nkb; ++kb) {
      mbar_wait(full_bar(stage), phase);
      tc_fence_after();
      const uint32_t sa = smem_base + stage * stage_bytes;
      const uint64_t wdesc = make_sdesc_k_sw128(sa);
      if (elect_one()) {
        for (int c = 0; c < chunks; ++c) {
          const uint64_t xdesc = make_sdesc_k_sw128(sa + kATile + c * chunk * 128);
#pragma unroll
          for (int k = 0; k < kKb / 16; ++k) umma_f16(tmem_base + c * chunk, wdesc + 2 * k, xdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(empty_bar(stage));
        if (kb == nkb - 1) umma_commit(done_bar);
      }
      __syncwarp();
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
  } else {
    if (warp <= kProducers) produce(warp - 1);
    // accumulator -> exchange tile over the stages (every TMA byte and every MMA operand in them has been consumed by then)
    const int q = warp & 3, half = (warp - 2) >> 2;
    mbar_wait(done_bar, 0);
    tc_fence_after();
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const int valid = min(args.tile_tokens, t_end - t0);
    for (int c = half * 16; c < valid; c += 32) {
      uint32_t r[16];
      tmem_ld16(taddr + c, r);
      tmem_ld_wait();
      const uint32_t dst = smem_base + (c * kFeat + q * 32 + lane) * 4;
#pragma unroll
      for (int i = 0; i < 16; ++i) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + i * kFeat * 4), "r"(r[i]) : "memory");
    }
    tc_fence_before();
  }
  if (SPLIT) cluster_sync_all(); else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, cols);
  }
  if (warp >= 2) {
    if (!GROUPED) griddep_wait();  // residual and output may belong to kernels before
    const int et = threadIdx.x - 64;
    const int share = (args.tile_tokens + S - 1) / S, lo = rank * share;
    const int hi = min(min(args.tile_tokens, lo + share), t_end - t0);
    const float scale = args.scale;
    if (args.mode == PG_EPI_GEGLU) {
      // rows of a weight tile: [64 gate | 64 up]; half a warp takes the 64 outputs of one token
      const int c = (et & 15) * 4, fo = f0 / 2 + c;
      float4 bg = make_float4(0.f, 0.f, 0.f, 0.f), bu = bg;
      if (args.bias != nullptr) {
        bg = *reinterpret_cast<const float4*>(args.bias + f0 + c);
        bu = *reinterpret_cast<const float4*>(args.bias + f0 + 64 + c);
      }
      auto unit = [&](auto kind) {
        for (int t = lo + (et >> 4); t < hi; t += 16 * kU) {
          float4 g[kU], u[kU];
#pragma unroll
          for (int j = 0; j < kU; ++j) {
            const uint32_t row = smem_base + (min(t + 16 * j, hi - 1) * kFeat + c) * 4;
            g[j] = gather4<SPLIT>(row, S);
            u[j] = gather4<SPLIT>(row + 256, S);
          }
#pragma unroll
          for (int j = 0; j < kU; ++j) {
            if (t + 16 * j >= hi) break;
            uint2 o;
            o.x = pack_bf16(glu_act(g[j].x + bg.x, u[j].x + bu.x, decltype(kind)::value, scale, args.glu_alpha), glu_act(g[j].y + bg.y, u[j].y + bu.y, decltype(kind)::value, scale, args.glu_alpha));
            o.y = pack_bf16(glu_act(g[j].z + bg.z, u[j].z + bu.z, decltype(kind)::value, scale, args.glu_alpha), glu_act(g[j].w + bg.w, u[j].w + bu.w, decltype(kind)::value, scale, args.glu_alpha));
            *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(args.out) + static_cast<long long>(t0 + t + 16 * j) * args.ldo + fo) = o;
          }
        }
      };
      with_glu(args.act, unit);
    } else {
      const int c = (et & 31) * 4, f = f0 + c;
      if (f < args.features) {  // (host: features % 4 == 0)
        float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (args.bias != nullptr) {
          b = *reinterpret_cast<const float4*>(args.bias + f);
          b.x *= scale; b.y *= scale; b.z *= scale; b.w *= scale;
        }
        auto rows = [&](auto act) {
          for (int t = lo + (et >> 5); t < hi; t += 8 * kU) {
            // the residual rows of kU tokens are under way before the first is needed
            float4 v[kU], h[kU];
            float* o[kU];
#pragma unroll
            for (int j = 0; j < kU; ++j) {
              const long long tok = t0 + min(t + 8 * j, hi - 1);
              h[j] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (args.mode != PG_EPI_BF16) {
                o[j] = static_cast<float*>(args.out) + (args.out_row_map != nullptr ? static_cast<long long>(__ldg(args.out_row_map + tok)) : tok) * args.ldo + f;
                if (args.resid != nullptr)
                  h[j] = *reinterpret_cast<const float4*>(args.resid + (args.resid_mod > 0 ? tok % args.resid_mod : tok) * args.ldr + f);
              }
            }
#pragma unroll
            for (int j = 0; j < kU; ++j) v[j] = gather4<SPLIT>(smem_base + (min(t + 8 * j, hi - 1) * kFeat + c) * 4, S);
#pragma unroll
            for (int j = 0; j < kU; ++j) {
              if (t + 8 * j >= hi) break;
              v[j].x = fmaf(v[j].x, scale, b.x); v[j].y = fmaf(v[j].y, scale, b.y); v[j].z = fmaf(v[j].z, scale, b.z); v[j].w = fmaf(v[j].w, scale, b.w);
              if (GROUPED && decltype(act)::value == 3) {  // neighbouring features are a gate and its up value
                *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(args.out) + static_cast<long long>(t0 + t + 8 * j) * args.ldo + f / 2) =
                    pack_bf16(v[j].x / (1.0f + expf(-v[j].x)) * v[j].y, v[j].z / (1.0f + expf(-v[j].z)) * v[j].w);
              } else if (args.mode == PG_EPI_BF16) {
                if (decltype(act)::value) {
                  v[j].x = epilogue_act(v[j].x, decltype(act)::value); v[j].y = epilogue_act(v[j].y, decltype(act)::value);
                  v[j].z = epilogue_act(v[j].z, decltype(act)::value); v[j].w = epilogue_act(v[j].w, decltype(act)::value);
                }
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(args.out) + static_cast<long long>(t0 + t + 8 * j) * args.ldo + f) =
                    make_uint2(pack_bf16(v[j].x, v[j].y), pack_bf16(v[j].z, v[j].w));
              } else {
                *reinterpret_cast<float4*>(o[j]) = make_float4(v[j].x + h[j].x, v[j].y + h[j].y, v[j].z + h[j].z, v[j].w + h[j].w);
              }
            }
          }
        };
        if (GROUPED && args.act == 3) rows(ActConst<3>{});
        else with_act(args.mode == PG_EPI_BF16 ? args.act : 0, rows);
      }
    }
  }
  if (SPLIT) cluster_sync_all();  // nobody leaves while a peer reads its exchange tile
}

bool configure() {
  static bool configured[kMaxDevices] = {};
  const int dev = current_device();
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(gemm_cluster_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax + 256) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_cluster_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax + 256) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_cluster_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax + 256) != cudaSuccess) {
      cudaGetLastError();  // do not leave a sticky error behind
      return false;
    }
    configured[dev] = true;
  }
  return true;
}

// Clusters of S CTAs that the device holds at once (a cluster lives in one GPC: at 1 CTA per SM, B200 holds 74 of 2, 45 of 3, 33 of 4, 22 of 6, 15 of 8).
int clusters_at_once(int S) {
  static int known[kMaxDevices][kMaxSplit + 1] = {};
  const int dev = current_device();
  if (known[dev][S] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemMax + 256;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (!configure() || cudaOccupancyMaxActiveClusters(&n, gemm_cluster_kernel<true>, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = num_sms() / (S + 1) > 0 ? num_sms() / (S + 1) : 1;
    }
    known[dev][S] = n;
  }
  return known[dev][S];
}

}  // namespace

ClusterGemmPlan plan_cluster_gemm(int tokens, int features, int K) {
  // A plan is the same for every token count of a step of 16 (tiles are multiples of 16), and a thread keeps those that it made.  (Where every call brings another
  // count -- prompts, the runs of routed experts -- a search per launch, which asked the driver for the device in every turn, made it 6.8 us of host time instead of 5.3.)
  tokens = (tokens + 15) / 16 * 16;
  struct Known { int dev, tokens, features, K; ClusterGemmPlan plan; };
  static thread_local Known known[512] = {};
  const int dev = current_device();
  Known& slot = known[(static_cast<unsigned>(tokens / 16) * 0x9E3779B1u ^ static_cast<unsigned>(features) * 0x85EBCA77u ^ static_cast<unsigned>(K) * 0xC2B2AE3Du) >> 23];
  if (slot.tokens == tokens && slot.features == features && slot.K == K && slot.dev == dev) return slot.plan;
  int at_once[kMaxSplit + 1];
  for (int S = 1; S <= kMaxSplit; S = S < 4 ? S + 1 : S + 2) at_once[S] = S == 1 ? num_sms() : clusters_at_once(S);
  ClusterGemmPlan best{0, 0, 0, 0.f};
  const int f_tiles = (features + kFeat - 1) / kFeat, total_kb = (K + kKb - 1) / kKb;
  for (int nt = (tokens + 383) / 384; nt <= (tokens + 383) / 384 + 7; ++nt) {
    int tile = (tokens + nt - 1) / nt;
    tile = tile > 256 ? (tile + 31) / 32 * 32 : (tile + 15) / 16 * 16;
    if (best.split != 0 && tile < 32) break;
    for (int S = 1; S <= kMaxSplit && S <= total_kb; S = S < 4 ? S + 1 : S + 2) {
      const int per = (total_kb + S - 1) / S;
      if ((total_kb + per - 1) / per != S) continue;  // a rank without work
      const int waves = (f_tiles * nt + at_once[S] - 1) / at_once[S];
      // clocks: launch, dependency wait and first bytes; an SM takes in 64 bytes a clock; the exchange writes and reads its tile
      const float cost = waves * (4000.f + per * (256.f + 2.f * tile) + (S > 1 ? 1500.f + 16.f * tile : 10.f * tile));
      if (best.split == 0 || cost < best.clocks) best = ClusterGemmPlan{tile, S, waves, cost};
    }
  }
  slot = Known{dev, tokens, features, K, best};
  return best;
}

int launch_cluster_gemm(const ClusterGemmPlan& plan, const void* x, long long ldx, const void* w, long long ldw, ClusterGemmArgs a, cudaStream_t st) {
  a.tile_tokens = plan.tile_tokens;
  a.split = plan.split;
  const int stage = kATile + a.tile_tokens * 128, exchange = a.tile_tokens * kFeat * 4;
  a.stages = kSmemMax / stage < 8 ? kSmemMax / stage : 8;
  const int per = ((a.K + kKb - 1) / kKb + a.split - 1) / a.split;
  if (a.stages > per) a.stages = per < 2 ? 2 : per;
  const int tiles = a.stages * stage > exchange ? a.stages * stage : exchange;
  a.smem_tiles = (tiles + 1023) / 1024 * 1024;
  if (a.smem_tiles > kSmemMax || !configure()) return PG_ERR_CUDA;
  CUtensorMap tw, tx;
  int rc;
  if ((rc = make_tmap_2d(&tw, w, a.features, a.K, ldw, kFeat)) != PG_OK) return rc;
  if ((rc = make_tmap_2d(&tx, x, a.tokens, a.K, ldx, a.tile_tokens > 256 ? a.tile_tokens / 2 : a.tile_tokens)) != PG_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.features + kFeat - 1) / kFeat * a.split, (a.tokens + a.tile_tokens - 1) / a.tile_tokens);
  cfg.blockDim = dim3(kThreads);
  if (a.tile_tokens > 256 && a.smem_tiles + 256 < kClusterSmemWide) return PG_ERR_ARG;  // (never: such tiles come in steps of 32 tokens)
  cfg.dynamicSmemBytes = a.split > 1 && a.smem_tiles + 256 < kClusterSmemAlone ? kClusterSmemAlone : a.smem_tiles + 256;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = a.split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pg_pdl_enabled() ? 2 : 1;
  pg_count_launch(1);
  return cudaLaunchKernelEx(&cfg, a.split > 1 ? gemm_cluster_kernel<true> : gemm_cluster_kernel<false>, tw, tx, a) == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}

int launch_grouped_gemm(const void* x, int rows, int K, const void* w, int experts, int F, void* out, bool out_f32, int act, const int* plan, int max_tiles,
                        int most_rows, cudaStream_t st) {
  if (!configure() || max_tiles <= 0 || max_tiles > 65535) return PG_ERR_CUDA;
  ClusterGemmArgs a = {};
  a.tokens = rows; a.features = F; a.K = K; a.mode = out_f32 ? PG_EPI_F32 : PG_EPI_BF16; a.act = act; a.scale = 1.f; a.out = out; a.plan = plan;
  a.ldo = act == 3 ? F / 2 : F;
  a.split = 1;
  a.tile_tokens = most_rows >= 64 ? 64 : (most_rows + 15) / 16 * 16;  // (the plan's tiles hold up to 64 rows)
  // two CTAs per SM: tiles are short and their number is known to the device only
  const int stage = kATile + a.tile_tokens * 128, per = (K + kKb - 1) / kKb;
  a.stages = 104 * 1024 / stage < 8 ? 104 * 1024 / stage : 8;
  if (a.stages > per) a.stages = per < 2 ? 2 : per;
  const int exchange = a.tile_tokens * kFeat * 4, tiles = a.stages * stage > exchange ? a.stages * stage : exchange;
  a.smem_tiles = (tiles + 1023) / 1024 * 1024;
  CUtensorMap tw, tx;
  int rc;
  if ((rc = make_tmap_2d(&tw, w, static_cast<long long>(experts) * F, K, K, kFeat)) != PG_OK) return rc;
  if ((rc = make_tmap_2d(&tx, x, rows, K, K, a.tile_tokens)) != PG_OK) return rc;
  return launch_kernel(gemm_cluster_kernel<false, true>, dim3((F + kFeat - 1) / kFeat, max_tiles), dim3(kThreads), a.smem_tiles + 256, st, tw, tx, a) == cudaSuccess
             ? PG_OK : PG_ERR_CUDA;
}

}  // namespace pg
