// Causal attention of prompt portions over the paged bf16 cache on the 5th-generation tensor cores, fp32 probabilities kept (the design notes of
// seq_attention_mma.cu hold: P is cut into three bf16 terms exactly, P V is three passes).  This kernel takes what prompts usually are -- pages of 64 keys (or a
// multiple, or 8, 16, 32), softmax scores with nothing but scale, soft cap, window and kept first keys -- and leaves logistic weights, distance penalties and other
// page sizes to that one.
//
// CTA = 128 query rows (token x query head of one k/v head) of one entry, keys in tiles of 64, two CTAs per SM.  Warp 0 brings pages in by TMA, warp 1 issues
// every tcgen05.mma, warps 2 .. 5 are the softmax, a thread per query row:
//   * S = Q K^T: 128 x 64 into tensor memory; a thread reads its row of 64 scores, masks, exponentiates -- no exchange between lanes, the row sum is its own;
//   * P goes back to tensor memory as three 32-column bf16 tiles and is the A operand of P V from there (12 instructions a tile): it never passes through shared memory;
//   * P lies over its own S (read by then) and 32 columns more, and there are two such areas (values 64 wide; for 128 the 256 columns of a CTA leave room for one): the next
//     tile's S is multiplied while this tile's exponentials run, and no tile waits for P V of the one before unless it rescales O.  So a warp cuts one piece of a row
//     (logic pipe) while the exponentials of the next are under way (MUFU);
//   * query rows come by TMA where a CTA has 128 of them and whole tokens, else with all of a thread's pieces requested together;
//   * O is rescaled only when a row's maximum grew by more than 2^8 (fp32 sums have the room);
//   * P V runs over all 128 rows with zero weights where a row does not see a key, and zero times a value that is not finite is no zero.  So a row whose sums are not finite is
//     computed again from the keys that it sees (row_from_visible_keys): a broken value reaches the rows that see it and no others.  (Rows that end or begin inside the loop
//     instead cost every prompt: 8 x 1024 tokens 140 -> 147 us; the check 142.)
// What bounds it: the softmax warps (MUFU 512 clocks a tile and warp, logic and permutes for the split 450, two warps on each pipe) and, with few tiles a CTA, its start (entry, page
// table, first tile: each a trip to memory).  Two threads a row share the same pipes, exponentials as polynomials on the FMA pipe cost more than they save.
// SPLIT: two CTAs of a cluster share a block's keys out, half of its tiles each, and the second hands its maxima, sums and O over through its shared memory, where the blocks are too few
// for the SMs (a portion of 128 tokens behind 1500, 32 blocks: 28 us, 21 so).
// us, mma.sync / here: 8 prompts of 897 .. 1024 tokens, 32 heads x 64 over 8 k/v heads 235 / 103; 2 portions of 333
// tokens behind 1400, 32 heads x 96 / 64: 144 / 49 (with P beside S, every tile waiting for P V of the one before, and query rows copied one piece after the other: 142 and 65;
// there a CTA of eight tiles spent 6500 of 31700 clocks before its first barrier).
#include <string.h>

#include "common.cuh"
#include "gemm_cluster.h"
#include "paligemma_b200.h"
#include "tmap.cuh"

using bf16 = __nv_bfloat16;

namespace pg {
namespace {

constexpr int kThreads = 192, kBox = 64 * 128;  // a box: 64 keys x 64 columns
constexpr float kLog2e = 1.4426950408889634f;

// D[tmem] (+)= A[tmem] * B[smem desc]: 128 x 16 bf16 A in 8 columns (two k values a column)
PG_DEVINL void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
PG_DEVINL void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
      "r"(r[14]), "r"(r[15])
      : "memory");
}
PG_DEVINL void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
               "r"(r[7])
               : "memory");
}
PG_DEVINL void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// MN-major operand as TMA lays it out ([k rows][64 columns], 128B swizzle); 64-column boxes `box` bytes apart
PG_DEVINL uint64_t make_sdesc_mn_sw128(uint32_t addr, uint32_t box) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((box >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

PG_DEVINL float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// as in seq_attention_mma.cu: tanh to fp32 accuracy, and the exact split by byte permutation
PG_DEVINL float tanh32(float x) {
  const float ax = fabsf(x), x2 = x * x;
  const float small = x * fmaf(x2, fmaf(x2, 0.13333333f, -0.33333334f), 1.0f);
  const float big = copysignf(1.0f - __fdividef(2.0f, ex2(ax * 2.885390082f) + 1.0f), x);
  return ax < 0.1f ? small : big;
}
PG_DEVINL void split3(uint64_t p, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  constexpr uint64_t minus = 0xbf800000bf800000ull;
  hi = __byte_perm(lo_of(p), hi_of(p), 0x7632);
  const uint64_t r = fma_pair(pair_of(lo_of(p) & 0xffff0000u, hi_of(p) & 0xffff0000u), minus, p);
  mid = __byte_perm(lo_of(r), hi_of(r), 0x7632);
  const uint64_t t = fma_pair(pair_of(lo_of(r) & 0xffff0000u, hi_of(r) & 0xffff0000u), minus, r);
  lo = __byte_perm(lo_of(t), hi_of(t), 0x7632);
}

template <int DIM, int VDIM>
struct Shape {
  static constexpr int KB = (DIM + 63) / 64, VB = VDIM / 64;     // 64-column boxes of a key / value tile
  static constexpr int Q_BYTES = KB * 128 * 128, KV_BYTES = (KB + VB) * kBox;
  static constexpr int STAGES = (112 * 1024 - Q_BYTES - 256) / KV_BYTES < 4 ? (112 * 1024 - Q_BYTES - 256) / KV_BYTES : 4;
  static constexpr int SMEM = Q_BYTES + STAGES * KV_BYTES + 256;
  static constexpr int NBUF = VDIM > 64 ? 1 : 2;                 // areas of 96 columns: S, then P over it
  static constexpr int COL_O = 96 * NBUF;
  // SPLIT holds its columns while it waits for its peer: it must not fit on an SM beside a split product that wants all 512 (gemm_cluster.h)
  static constexpr int SMEM_SPLIT = SMEM > 83 * 1024 ? SMEM : 83 * 1024;
  static_assert(COL_O + VDIM <= 256 && STAGES >= 2 && DIM % 16 == 0 && VDIM % 64 == 0 && 2 * (SMEM_SPLIT + kCtaShared) <= kSmShared, "two CTAs per SM");
  static_assert(SMEM_SPLIT + kClusterSmemWide + 2 * kCtaShared > kSmShared, "a split product's CTA of 512 columns would fit beside a shared block's");
};

// One query row by a warp, from the keys that it sees and no others: for rows whose sums are not finite (see above).  Scores, probabilities and sums in fp32; a lane has a key of
// 32 for the scores and VDIM / 32 columns of the values.
template <int DIM, int VDIM>
__device__ __noinline__ void row_from_visible_keys(const bf16* __restrict__ q, const bf16* __restrict__ k_pages, const bf16* __restrict__ v_pages, const int* __restrict__ pt, int page,
                                                   long long krow, long long vrow, int lim, int lo, int keep, float sc, float softcap, const float* sink, float out_scale,
                                                   const bf16* __restrict__ gate, int gate_per_head, bf16* __restrict__ out) {
  constexpr int NC = VDIM / 32;
  const int lane = threadIdx.x & 31;
  float m = -INFINITY, l = 0.f, acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = 0.f;
  for (int k0 = 0; k0 <= lim; k0 += 32) {
    if (k0 >= keep && k0 + 31 < lo) k0 = lo & ~31;
    const int j = k0 + lane;
    const bool vis = j <= lim && (j >= lo || j < keep);
    const unsigned seen = __ballot_sync(0xffffffffu, vis);
    const long long row = vis ? static_cast<long long>(pt[j / page]) * page + j % page : 0;
    float t = -INFINITY;
    if (vis) {
      float d = 0.f;
      for (int i = 0; i < DIM; ++i) d = fmaf(__bfloat162float(q[i]), __bfloat162float(k_pages[row * krow + i]), d);
      t = (softcap > 0.f ? softcap * tanh32(d * (sc / softcap)) : d * sc) * kLog2e;
    }
    float mx = t;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float mn = fmaxf(m, mx), off = mn > -INFINITY ? mn : 0.f, alpha = ex2(m - off), p = vis ? ex2(t - off) : 0.f;
    m = mn;
    l = l * alpha + p;
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] *= alpha;
    for (unsigned left = seen; left != 0; left &= left - 1) {
      const int src = __ffs(left) - 1;
      const float pj = __shfl_sync(0xffffffffu, p, src);
      const bf16* v = v_pages + __shfl_sync(0xffffffffu, row, src) * vrow + NC * lane;
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[c] = fmaf(pj, __bfloat162float(v[c]), acc[c]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  float osc = 1.f;
  if (sink != nullptr) {
    const float sk = *sink * kLog2e, mm = fmaxf(m, sk);
    osc = exp2f(m - mm);
    l = l * osc + exp2f(sk - mm);
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    float x = acc[c] * (osc / l * out_scale);
    if (gate != nullptr) x *= 1.0f / (1.0f + expf(-__bfloat162float(gate[gate_per_head ? 0 : NC * lane + c])));
    out[NC * lane + c] = __float2bfloat16_rn(x);
  }
}

template <int DIM, int VDIM, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 2) attn_ragged_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                     const __grid_constant__ CUtensorMap tmV,
                                                                     const bf16* __restrict__ q, const bf16* __restrict__ k_pages, const bf16* __restrict__ v_pages,
                                                                     const bf16* __restrict__ gate, long long ldg, bf16* __restrict__ out,
                                                                     const int* __restrict__ entry_row0, const int* __restrict__ entry_n, const int* __restrict__ entry_ctx,
                                                                     const int* __restrict__ page_table, int max_pages, int page, int H, int G, float scale, float softcap,
                                                                     int skip_single, int gate_per_head, int q_tma, int entries, int units, PgAttnScore sx) {
  using C = Shape<DIM, VDIM>;
  constexpr uint32_t IDESC_S = make_idesc_bf16(128, 64), IDESC_O = make_idesc_bf16(128, VDIM, 0, 1);
  griddep_wait();
  // The longest rows of all entries and heads come first (48 prompts of 193 .. 256 tokens, soft-capped: 243 us entry by entry, 198 so).  Where single tokens are left to another
  // kernel, the entries with rows are counted and numbered first, so that CTAs without any stand at the end and not between two blocks of rows; where the host has counted them (`units`)
  // there are none (2 portions + 40 singles, 192 CTAs with rows: 49 us, 60 with 3840 empty ones behind them, 71 with 2700 in front of the third block).
  const unsigned idx = SPLIT ? blockIdx.x / 2 : blockIdx.x, blocks = (SPLIT ? gridDim.x / 2 : gridDim.x) / static_cast<unsigned>(units * G);
  unsigned with_rows = entries;
  if (skip_single) {
    with_rows = 0;
    for (int i = 0; i < entries; i += 32) {
      const int at = i + static_cast<int>(lane_id());
      with_rows += __popc(__ballot_sync(0xffffffffu, at < entries && entry_n[at] != 1));
    }
  }
  if (idx >= blocks * with_rows * G) return;
  const unsigned unit = idx % (with_rows * G);
  int e = unit / G;
  if (skip_single) {
    int left = e;
    for (int i = 0;; i += 32) {
      const int at = i + static_cast<int>(lane_id());
      const unsigned here = __ballot_sync(0xffffffffu, at < entries && entry_n[at] != 1);
      if (left < __popc(here)) {
        e = i + __fns(here, 0, left + 1);
        break;
      }
      left -= __popc(here);
    }
  }
  const int g = unit % G, gsz = H / G;
  const int n = entry_n[e], ctx = entry_ctx[e], row0 = entry_row0[e];
  const int rows = n * gsz, r0 = static_cast<int>(blocks - 1 - idx / (with_rows * G)) * 128;
  if (r0 >= rows) return;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  if ((base & 1023u) != 0) __trap();
  const uint32_t kv0 = base + C::Q_BYTES, bar0 = kv0 + C::STAGES * C::KV_BYTES;
  auto kv_full = [&](int s) { return bar0 + 8u * s; };
  auto kv_empty = [&](int s) { return bar0 + 8u * (4 + s); };
  auto s_full = [&](int b) { return bar0 + 64u + 8u * b; };
  auto p_full = [&](int b) { return bar0 + 80u + 8u * b; };
  auto o_done = [&](int b) { return bar0 + 96u + 8u * b; };  // (two: with one, a wait for tile j - 1 would pass while j - 2 is still under way)
  const uint32_t q_full = bar0 + 112, tmem_slot = bar0 + 120;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool by_tma = q_tma && r0 + 128 <= rows;  // (rows past the entry's may lie past the end of q)
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(kv_full(s), 1);
      mbar_init(kv_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(s_full(b), 1);
      mbar_init(p_full(b), 4);
      mbar_init(o_done(b), 1);
    }
    mbar_init(q_full, 1);
    mbar_fence_init();
    if (by_tma) {
      mbar_expect_tx(q_full, C::Q_BYTES);
#pragma unroll
      for (int b = 0; b < C::KB; ++b) tma_load_3d(base + b * (128 * 128), &tmQ, q_full, 64 * b, g * gsz, row0 + r0 / gsz, kEvictNormal);
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  if (!by_tma) {  // query rows, swizzled as TMA would lay them (zeros past the end and past DIM)
    constexpr int N = (128 * C::KB * 8 + kThreads - 1) / kThreads;
    uint4 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int id = threadIdx.x + i * kThreads, r = id / (C::KB * 8), cc = id % (C::KB * 8), rr = r0 + r;
      v[i] = make_uint4(0, 0, 0, 0);
      if (r < 128 && rr < rows && cc * 8 < DIM)
        v[i] = *reinterpret_cast<const uint4*>(q + static_cast<long long>(row0 + rr / gsz) * (static_cast<long long>(H) * DIM) + static_cast<long long>(g * gsz + rr % gsz) * DIM + cc * 8);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int id = threadIdx.x + i * kThreads, r = id / (C::KB * 8), cc = id % (C::KB * 8);
      if (r < 128)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(base + (cc >> 3) * (128 * 128) + r * 128 + (((cc & 7) ^ (r & 7)) << 4)), "r"(v[i].x), "r"(v[i].y), "r"(v[i].z),
                     "r"(v[i].w) : "memory");
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");

  const int last_row = min(rows, r0 + 128) - 1, kmax = ctx + last_row / gsz;  // last key any row of the CTA sees
  const int window = sx.window > 0 ? sx.window : 0x3fffffff, keep = sx.window > 0 ? max(sx.keep_first, 0) : 0;
  const int keep_end = (keep + 63) & ~63, cta_lo = max(0, ctx + r0 / gsz - window + 1) & ~63;
  // key tiles wholly between the kept first keys and the first key inside the window of the CTA's first row are skipped
  const bool gap = cta_lo > keep_end;
  const int before = keep_end / 64, tiles = gap ? before + (kmax - cta_lo) / 64 + 1 : kmax / 64 + 1;
  auto key_of = [&](int i) { return gap && i >= before ? cta_lo + 64 * (i - before) : 64 * i; };
  const int rank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0, half = (tiles + 1) / 2;
  const int t0 = SPLIT && rank ? half : 0, t1 = SPLIT && !rank ? half : tiles;  // this CTA's tiles (the second of a cluster may have none)

  if (warp == 0) {
    if (lane == 0) {
      const int* pt = page_table + static_cast<long long>(e) * max_pages;
      int stage = 0;
      uint32_t phase = 0;
      const int piece = min(page, 64);  // rows of a box: a tile is (part of) a page, or several pages (those past the last key are left out)
      auto row_at = [&](int key) { return pt[key / page] * page + key % page; };
      int first = t0 < t1 ? row_at(key_of(t0)) : 0;
      for (int i = t0; i < t1; ++i) {
        const int k0 = key_of(i), pieces = min(64, kmax + 1 - k0 + piece - 1) / piece;
        int row = first;
        if (i + 1 < t1) first = row_at(key_of(i + 1));
        const uint32_t sk = kv0 + stage * C::KV_BYTES;
        mbar_wait(kv_empty(stage), phase ^ 1);
        mbar_expect_tx(kv_full(stage), (C::KB + C::VB) * 128 * piece * pieces);
        for (int part = 0; part < pieces; ++part) {
          if (part > 0) row = row_at(k0 + part * piece);
          const uint32_t dst = sk + part * piece * 128;
#pragma unroll
          for (int b = 0; b < C::KB; ++b) tma_load_2d(dst + b * kBox, &tmK, kv_full(stage), g * DIM + 64 * b, row, kEvictNormal);
#pragma unroll
          for (int b = 0; b < C::VB; ++b) tma_load_2d(dst + (C::KB + b) * kBox, &tmV, kv_full(stage), g * VDIM + 64 * b, row, kEvictNormal);
        }
        if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // tile j: S in area j % NBUF, its P over it; S of tile j + NBUF behind P V of tile j, whose area it takes (one thread's products run in order)
    int stage = 0, ahead = 0, js = 0;  // stages of P V and of S; number of the next S
    uint32_t ahead_phase = 0;
    auto issue_s = [&]() {
      mbar_wait(kv_full(ahead), ahead_phase);
      tc_fence_after();
      const uint32_t sk = kv0 + ahead * C::KV_BYTES, to = tmem + 96 * (js % C::NBUF);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < DIM / 16; ++k)
          umma_f16(to, make_sdesc_k_sw128(base + (k >> 2) * (128 * 128)) + 2 * (k & 3), make_sdesc_k_sw128(sk + (k >> 2) * kBox) + 2 * (k & 3), IDESC_S, k > 0 ? 1u : 0u);
        umma_commit(s_full(js % C::NBUF));
      }
      __syncwarp();
      if (++ahead == C::STAGES) { ahead = 0; ahead_phase ^= 1; }
      ++js;
    };
    if (by_tma) mbar_wait(q_full, 0);
    for (int b = 0; b < C::NBUF; ++b)
      if (t0 + js < t1) issue_s();
    for (int j = 0; t0 + j < t1; ++j) {
      const int k0 = key_of(t0 + j);
      const uint32_t sv = kv0 + stage * C::KV_BYTES + C::KB * kBox, area = tmem + 96 * (j % C::NBUF);
      if (k0 + 63 > kmax) {  // the last tile: keys nobody sees weigh zero, whatever lies there
        for (int r = kmax + 1 - k0 + lane; r < 64; r += 32)
#pragma unroll
          for (int b = 0; b < C::VB; ++b)
#pragma unroll
            for (int c = 0; c < 8; ++c) asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(sv + b * kBox + r * 128 + c * 16), "r"(0) : "memory");
        fence_proxy_async_smem();
        __syncwarp();
      }
      mbar_wait(p_full(j & 1), (j >> 1) & 1);
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int term = 0; term < 3; ++term)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16_ts(tmem + C::COL_O, area + term * 32 + k * 8, make_sdesc_mn_sw128(sv + k * 2048, kBox), IDESC_O, (j > 0 || term > 0 || k > 0) ? 1u : 0u);
        umma_commit(kv_empty(stage));
        umma_commit(o_done(j & 1));
      }
      __syncwarp();
      if (t0 + js < t1) issue_s();
      if (++stage == C::STAGES) stage = 0;
    }
  } else {
    const int qd = warp & 3, r = qd * 32 + lane, rr = r0 + r;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(qd * 32) << 16);
    const bool there = rr < rows;
    const int head = g * gsz + (there ? rr % gsz : 0);
    const int lim = there ? ctx + rr / gsz : -1, lo = lim - window + 1;  // last and first key of the row's window
    // keys of a tile that every row of the warp sees: up to the first row's position, from the last row's window on
    const int wr = r0 + qd * 32;
    const bool warp_whole = wr + 32 <= rows;
    const int all_lim = ctx + wr / gsz, all_lo = ctx + (wr + 31) / gsz - window + 1;
    const float sc = scale * (sx.head_scale != nullptr ? sx.head_scale[head] : 1.f);
    const bool plain = !(softcap > 0.f) && sx.head_scale == nullptr && scale > 0.f;  // the maximum commutes with the scale, which rides on the exponent's FMA
    const float unit = plain ? scale * kLog2e : kLog2e, in = softcap > 0.f ? sc / softcap : 0.f;
    float m = -INFINITY, l = 0.f;
    int j = 0;
    for (; t0 + j < t1; ++j) {
      const int k0 = key_of(t0 + j);
      const uint32_t area = lanes + 96 * (j % C::NBUF);
      mbar_wait(s_full(j % C::NBUF), (j / C::NBUF) & 1);
      tc_fence_after();
      float s[64];
      {
        uint32_t v[4][16];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld16(area + 16 * c, v[c]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 64; ++i) s[i] = __uint_as_float(v[i >> 4][i & 15]);
      }
      if (!plain) {
        if (softcap > 0.f) {
#pragma unroll
          for (int i = 0; i < 64; ++i) s[i] = softcap * tanh32(s[i] * in);
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) s[i] *= sc;
        }
      }
      if (!(warp_whole && k0 + 63 <= all_lim && (k0 >= all_lo || k0 + 64 <= keep))) {
        const int hi = lim - k0, lw = lo - k0, kp = keep - k0;
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (!(i <= hi && (i >= lw || i < kp))) s[i] = -INFINITY;
      }
      float mx;
      {
        float m8[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) m8[i] = s[i];
#pragma unroll
        for (int i = 8; i < 56; i += 16)
#pragma unroll
          for (int k = 0; k < 8; ++k) m8[k] = max3(m8[k], s[i + k], s[i + 8 + k]);
#pragma unroll
        for (int k = 0; k < 8; ++k) m8[k] = fmaxf(m8[k], s[56 + k]);
        mx = max3(max3(m8[0], m8[1], m8[2]), max3(m8[3], m8[4], m8[5]), fmaxf(m8[6], m8[7])) * unit;
      }
      const bool need = mx > m + 8.0f;  // (from -inf: every finite maximum)
      const float mn = need ? mx : m;
      const float alpha = need ? ex2(m - mn) : 1.0f, off = mn > -INFINITY ? -mn : 0.f;  // rows that see no key yet weigh nothing
      m = mn;
      if (__any_sync(0xffffffffu, need) && j > 0) {
        mbar_wait(o_done((j - 1) & 1), ((j - 1) >> 1) & 1);  // P V of the tile before
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < VDIM; c += 16) {
          uint32_t v[16];
          tmem_ld16(lanes + C::COL_O + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
          tmem_st16(lanes + C::COL_O + c, v);
        }
      }
      // pieces of 16 scores: the exponentials of a piece are requested before the piece in front is cut and stored
      uint64_t s2[2] = {0, 0}, pp[2][8];
      const uint64_t unit2 = pair_of(unit, unit), off2 = pair_of(off, off);
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        if (c < 4) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int at = (16 * c + 2 * i) & 63;
            const uint64_t x = fma_pair(pair_of(s[at], s[at + 1]), unit2, off2);
            pp[c & 1][i] = pair_of(ex2(lo_f32(x)), ex2(hi_f32(x)));
          }
        }
        if (c > 0) {
          uint32_t hi[8], mid[8], low[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t p = pp[(c - 1) & 1][i];
            s2[i & 1] = add_pair(s2[i & 1], p);
            split3(p, hi[i], mid[i], low[i]);
          }
          tmem_st8(area + 8 * (c - 1), hi);
          tmem_st8(area + 32 + 8 * (c - 1), mid);
          tmem_st8(area + 64 + 8 * (c - 1), low);
        }
      }
      s2[0] = add_pair(s2[0], s2[1]);
      l = l * alpha + (lo_f32(s2[0]) + hi_f32(s2[0]));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full(j & 1));
    }
    if (!SPLIT || j > 0) {
      mbar_wait(o_done((j - 1) & 1), ((j - 1) >> 1) & 1);
      tc_fence_after();
    }
    // SPLIT: the second CTA's maxima, sums and O of its 128 rows lie over its key tiles, [4 columns][row] and then [2][row]
    float own = 1.f, other = 0.f;  // factors of this CTA's and the other's sums
    uint32_t far = 0;
    if constexpr (SPLIT) {
      const uint32_t at = kv0 + r * 16, tail = kv0 + VDIM * 128 * 4 + r * 4;
      if (rank == 1) {
#pragma unroll 1
        for (int c = 0; c < VDIM; c += 16) {
          uint32_t v[16] = {};
          if (j > 0) {
            tmem_ld16(lanes + C::COL_O + c, v);
            tmem_ld_wait();
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + (c / 4 + i) * 2048), "r"(v[4 * i]), "r"(v[4 * i + 1]), "r"(v[4 * i + 2]), "r"(v[4 * i + 3]) : "memory");
        }
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(tail), "f"(m) : "memory");
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(tail + 512), "f"(l) : "memory");
      }
      cluster_sync_all();
      if (rank == 0) {
        uint32_t there_m;
        float m2, l2;
        asm volatile("mapa.shared::cluster.u32 %0, %1, 1;" : "=r"(far) : "r"(at));
        asm volatile("mapa.shared::cluster.u32 %0, %1, 1;" : "=r"(there_m) : "r"(tail));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(m2) : "r"(there_m) : "memory");
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(l2) : "r"(there_m + 512) : "memory");
        const float mm = fmaxf(m, m2);
        own = ex2(m - mm);
        other = ex2(m2 - mm);  // no key seen there: 0
        l = l * own + l2 * other;
        m = mm;
      }
    }
    if (!SPLIT || rank == 0) {
      float osc = 1.f;
      if (sx.sink != nullptr) {  // the sink joins the denominator once (m is in base-2 units)
        const float sk = sx.sink[head] * kLog2e, mm = fmaxf(m, sk);
        osc = exp2f(m - mm);
        l = l * osc + exp2f(sk - mm);
      }
      const float inv = osc / l * (sx.out_scale != 0.f ? sx.out_scale : 1.f);
      const long long t = row0 + (there ? rr / gsz : 0), ldo = sx.out_ld > 0 ? sx.out_ld : static_cast<long long>(H) * VDIM;
      bf16* o = out + t * ldo + static_cast<long long>(head) * VDIM;
      const bf16* gt = gate == nullptr ? nullptr : gate + t * ldg + (gate_per_head ? static_cast<long long>(head) : static_cast<long long>(head) * VDIM);
      bool odd = false;  // a sum of the row is not finite
      const float gh = gate != nullptr && gate_per_head ? 1.0f / (1.0f + expf(-__bfloat162float(*gt))) : 1.f;
#pragma unroll 1
      for (int c0 = 0; c0 < VDIM; c0 += 64) {
        uint32_t all[4][16];
#pragma unroll
        for (int i = 0; i < 4; ++i) tmem_ld16(lanes + C::COL_O + c0 + 16 * i, all[i]);
        tmem_ld_wait();
        if constexpr (SPLIT) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float4 o2;
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o2.x), "=f"(o2.y), "=f"(o2.z), "=f"(o2.w) : "r"(far + (c0 / 4 + i) * 2048) : "memory");
            uint32_t* v = &all[i / 4][i % 4 * 4];
            v[0] = __float_as_uint(fmaf(__uint_as_float(v[0]), own, o2.x * other));
            v[1] = __float_as_uint(fmaf(__uint_as_float(v[1]), own, o2.y * other));
            v[2] = __float_as_uint(fmaf(__uint_as_float(v[2]), own, o2.z * other));
            v[3] = __float_as_uint(fmaf(__uint_as_float(v[3]), own, o2.w * other));
          }
        }
#pragma unroll
        for (int part = 0; part < 4; ++part) {
          if (!there) break;
          const int c = c0 + 16 * part;
          const uint32_t(&v)[16] = all[part];
          float x[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            odd = odd || (v[i] & 0x7f800000u) == 0x7f800000u;
            x[i] = __uint_as_float(v[i]) * inv;
          }
          if (gate != nullptr) {
            if (gate_per_head) {
#pragma unroll
              for (int i = 0; i < 16; ++i) x[i] *= gh;
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float2 gg = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(gt + c)[i]);
                x[2 * i] *= 1.0f / (1.0f + expf(-gg.x));
                x[2 * i + 1] *= 1.0f / (1.0f + expf(-gg.y));
              }
            }
          }
          uint4* d = reinterpret_cast<uint4*>(o + c);
          d[0] = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
          d[1] = make_uint4(pack_bf16(x[8], x[9]), pack_bf16(x[10], x[11]), pack_bf16(x[12], x[13]), pack_bf16(x[14], x[15]));
        }
        __syncwarp();
      }
      for (unsigned left = __ballot_sync(0xffffffffu, odd); left != 0; left &= left - 1) {
        const int row = r0 + qd * 32 + __ffs(left) - 1, hd = g * gsz + row % gsz, last = ctx + row / gsz;
        const long long tk = row0 + row / gsz;
        row_from_visible_keys<DIM, VDIM>(q + (tk * H + hd) * DIM, k_pages + static_cast<long long>(g) * DIM, v_pages + static_cast<long long>(g) * VDIM,
                                         page_table + static_cast<long long>(e) * max_pages, page, static_cast<long long>(G) * DIM, static_cast<long long>(G) * VDIM, last, last - window + 1, keep,
                                         scale * (sx.head_scale != nullptr ? sx.head_scale[hd] : 1.f), softcap, sx.sink != nullptr ? sx.sink + hd : nullptr,
                                         sx.out_scale != 0.f ? sx.out_scale : 1.f,
                                         gate == nullptr ? nullptr : gate + tk * ldg + (gate_per_head ? static_cast<long long>(hd) : static_cast<long long>(hd) * VDIM), gate_per_head,
                                         out + tk * ldo + static_cast<long long>(hd) * VDIM);
      }
    }
    tc_fence_before();
  }
  if constexpr (SPLIT) {
    if (warp < 2) cluster_sync_all();  // the second CTA's sums are there
    cluster_sync_all();                // and have been read
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

template <int DIM, int VDIM, bool SPLIT>
int launch(const void* q, const void* kp, const void* vp, const void* gate, long long ldg, void* out, const int* row0, const int* n, const int* ctx, const int* pt,
           int max_pages, int page, int entries, int units, int max_n, int H, int G, float scale, float softcap, int skip_single, int gate_per_head, const PgAttnScore& sx,
           cudaStream_t st) {
  using C = Shape<DIM, VDIM>;
  constexpr int smem = SPLIT ? C::SMEM_SPLIT : C::SMEM;
  const long long ctas = (static_cast<long long>(max_n) * (H / G) + 127) / 128 * G * units;
  if ((SPLIT ? 2 * ctas : ctas) > 0x7fffffff) return 1;
  static bool configured[kMaxDevices] = {};
  const int dev = current_device();
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(attn_ragged_tc_kernel<DIM, VDIM, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return PG_ERR_CUDA;
    }
    configured[dev] = true;
  }
  const int gsz = H / G;
  // query rows of whole tokens: boxes of [128 / gsz tokens][gsz heads][64 columns]; only rows of the step are read, so the token count is a bound and not a size
  const int q_tma = 128 % gsz == 0;
  CUtensorMap tq;
  if (q_tma) {
    const int rcq = make_tmap_rows3(&tq, q, DIM, H, 1LL << 24, gsz, 128 / gsz);
    if (rcq != PG_OK) return rcq;
  } else {
    memset(&tq, 0, sizeof(tq));
  }
  // the pools as matrices of rows: only pages named by the table are read, so the row count is a bound and not a size
  CUtensorMap tk, tv;
  int rc;
  if ((rc = make_tmap_2d(&tk, kp, 1LL << 30, static_cast<long long>(G) * DIM, static_cast<long long>(G) * DIM, page < 64 ? page : 64)) != PG_OK) return rc;
  if ((rc = make_tmap_2d(&tv, vp, 1LL << 30, static_cast<long long>(G) * VDIM, static_cast<long long>(G) * VDIM, page < 64 ? page : 64)) != PG_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(SPLIT ? 2 * ctas : ctas));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = SPLIT ? 1 : 0;  // (behind the whole of the kernel before, as launch_spread)
  cudaLaunchKernelEx(&cfg, attn_ragged_tc_kernel<DIM, VDIM, SPLIT>, tq, tk, tv, static_cast<const bf16*>(q), static_cast<const bf16*>(kp), static_cast<const bf16*>(vp),
                     static_cast<const bf16*>(gate), ldg, static_cast<bf16*>(out), row0, n, ctx, pt, max_pages, page, H, G, scale, softcap, skip_single, gate_per_head, q_tma, entries, units, sx);
  pg_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}

}  // namespace
}  // namespace pg

// Launches the call when it is one of this file's (PG_OK or an error), else returns 1.  Everything that pg_attn_ragged_mma checks has been checked.
int pg_attn_ragged_tc(const void* q, const void* kp, const void* vp, const void* gate, long long ldg, void* out, const int* row0, const int* n, const int* ctx, const int* pt,
                      int max_pages, int page, int entries, int max_n, int H, int G, int dim, int vdim, float scale, float softcap, int skip_single, int gate_per_head,
                      int portions, int longest, const PgAttnScore& sx, cudaStream_t st) {
  // pages that a tile of 64 keys divides, or that divide it in whole swizzle rows
  if (!(page > 0 && (page % 64 == 0 || (page % 8 == 0 && 64 % page == 0))) || sx.logistic || sx.dist_a != nullptr || sx.out_ld % 8 != 0) return 1;
  // Blocks of 128 rows do not pay for a handful of rows in more CTAs than SMs (the mma.sync kernel's warps without rows idle; us, mma.sync / here, rows of a block x CTAs behind contexts of 1000:
  // 16 x 24 24.7 / 15.5, 16 x 96 24.9 / 21.5, 4 x 96 26.2 / 21.4, 4 x 192 28.8 / 33.4, 4 x 384 31.5 / 51.7; behind 500: 16 x 192 16.3 / 20.1, 8 x 320 17.8 / 29.6).  Entries without rows
  // for this kernel are no CTAs (`portions`, where the caller knows): 4 tokens behind 1000 beside 40 single ones, 32 heads over 8: 24.7 / 16.0.  Values of 128 columns leave one area for S
  // and P, so a few CTAs with short keys are as fast there (16 heads, mma.sync / here: 200 tokens 11.6 / 12.3, behind 500 25.6 / 22.4, 400 behind 2000 71 / 65).
  const int counted = portions > 0 && portions < entries ? portions : entries;
  const long long rows = static_cast<long long>(max_n) * (H / G), units = static_cast<long long>(G) * counted;
  if ((rows <= 16 && units > pg::num_sms()) || (dim == 64 && vdim == 128 && longest <= 256 && (rows + 63) / 64 * units <= pg::num_sms())) return 1;  // (longest 0: not known)
  // Two CTAs a block where the blocks are too few for the SMs and long enough to share out (portions and longest: entries with rows and the longest context with its new tokens, 0 where
  // the caller does not know; us, one CTA / two: 80 blocks of 24 .. 28 tiles 38 / 31, 32 of 24 .. 26 28 / 21, 64 of 16 40 / 35, 96 of 26 of 96 / 64 37 / 33; but 160 blocks of 24 .. 28
  // 40 / 41, 192 of 26 49 / 51, 128 of up to 8 15.6 / 16.5).
  const long long blocks = (rows + 127) / 128 * G * portions;
  const int reach = sx.window > 0 ? (longest < sx.window + (sx.keep_first > 0 ? sx.keep_first : 0) + 128 ? longest : sx.window + (sx.keep_first > 0 ? sx.keep_first : 0) + 128) : longest;
  const bool split = vdim == 64 && portions > 0 && 4 * blocks <= 3LL * pg::num_sms() && reach >= 12 * 64;
#define PG_TC1(D, V, S) return pg::launch<D, V, S>(q, kp, vp, gate, ldg, out, row0, n, ctx, pt, max_pages, page, entries, counted, max_n, H, G, scale, softcap, \
                                                   skip_single, gate_per_head, sx, st)
#define PG_TC(D, V)                  \
  if (dim == D && vdim == V) {       \
    if (V == 64 && split) PG_TC1(D, V, (V == 64)); \
    PG_TC1(D, V, false);             \
  }
  PG_TC(64, 64);
  PG_TC(96, 64);
  PG_TC(128, 128);
  PG_TC(64, 128);
  PG_TC(128, 64);
#undef PG_TC1
#undef PG_TC
  return 1;
}
