// The tcgen05 product for a moderate number of tokens (gemm_cluster.cu): what gemm_tcgen05.cu needs to choose and launch it.
#pragma once
#include <cuda_runtime.h>

namespace pg {

struct ClusterGemmArgs {
  int tokens, features, K;
  int mode, act;
  float scale, glu_alpha;
  void* out;
  long long ldo;
  const float* bias;
  const float* resid;
  long long ldr;
  const int* out_row_map;
  int resid_mod;
  const int* plan;  // grouped products: tiles (expert, first row, rows) from word 4 on, their number in word 0
  // set by the launcher
  int tile_tokens, split, stages, smem_tiles;
};

// tokens per tile, CTAs that share K, waves of the grid, and the estimated clocks of the launch
struct ClusterGemmPlan {
  int tile_tokens, split, waves;
  float clocks;
};

// Shared memory of CTAs that hold tensor memory while they wait for their cluster's peers.  Two clusters of two streams that met in opposite order on two SMs would wait for each other's
// columns for ever, so no two such CTAs whose columns are more than an SM's 512 may fit on one (228 KB; a CTA takes 1 KB beside its own):
//   * split products (gemm_cluster.cu) take more than half, so that two of them never share an SM;
//   * those of more than 256 tokens a tile hold all 512 columns and exchange kClusterWideTokens x 128 floats at least; shared prompt attention (seq_attention_tc.cu: 256 columns, two on
//     an SM) takes so much that it does not fit beside them;
//   * CTA pairs (gemm_tcgen05.cu) take all but a few KB.
constexpr int kSmShared = 228 * 1024, kCtaShared = 1024;
constexpr int kClusterSmemAlone = 114 * 1024, kClusterWideTokens = 288, kClusterSmemWide = kClusterWideTokens * 128 * 4 + 256;  // (barriers)
static_assert(2 * (kClusterSmemAlone + kCtaShared) > kSmShared, "two clustered CTAs would fit on one SM");

ClusterGemmPlan plan_cluster_gemm(int tokens, int features, int K);
int launch_cluster_gemm(const ClusterGemmPlan& plan, const void* x, long long ldx, const void* w, long long ldw, ClusterGemmArgs a, cudaStream_t st);

// One product per expert over its run of rows: out[r, :] = act(x[r, :] W_e^T) for the rows of every tile of `plan` (at most `max_tiles`, 64 rows each, and
// `most_rows` of them where that is fewer).
// w: [experts * F, K] dense; act 3: rows alternate gate / up, out has F / 2 columns; out bf16, or fp32 without activation.
int launch_grouped_gemm(const void* x, int rows, int K, const void* w, int experts, int F, void* out, bool out_f32, int act, const int* plan, int max_tiles,
                        int most_rows, cudaStream_t st);

}  // namespace pg
