// Whole runs of layers issued by one call: the launches of a SigLIP encoder or of a Gemma prompt pass are the same few per layer, and issuing each
// from Python costs 9 .. 13 us (argument checks, tensor metadata, the foreign call) where the launch itself costs 3 and the kernels of one
// image take 4 .. 10.  No kernels here.
#include <cmath>

#include "common.cuh"
#include "paligemma_b200.h"

bool pg_gemm_sums_once(int tokens, int features, int K, const void* out, long long ldo, const float* bias, int swap);  // gemm_tcgen05.cu

extern "C" int pg_weights_follow(int on) {
  if (!on && pg::t_weights_follow <= 0) return PG_ERR_ARG;  // (not given: taken back, it would silence the next one)
  pg::t_weights_follow += on ? 1 : -1;
  return PG_OK;
}

extern "C" int pg_gemm_residual(const void* x, long long ldx, const void* w, long long ldw, float* h, long long ldh, const float* bias, int tokens,
                                int features, int K, float scale, void* stream) {
  if (tokens <= 0 || features <= 0 || K <= 0) return PG_ERR_ARG;
  const int swap = tokens <= 128 ? 1 : 0, kb = (K + 63) / 64, sms = pg::num_sms();
  if (!swap && pg_gemm_sums_once(tokens, features, K, h, ldh, bias, 0))
    return pg_gemm_bf16(x, ldx, w, ldw, h, ldh, bias, h, ldh, tokens, features, K, PG_EPI_F32, 0, scale, 0, 1, stream);
  // what is left: decode steps, many tokens, and rows off a 16-byte boundary
  int tiles;
  if (swap) {
    tiles = (features + 127) / 128;
  } else if (kb < 128) {
    // short and medium K: count 128 x 64 tiles -- the kernel narrows its N tile before K is split, because every split costs a full
    // fp32 red.add pass over the output tile
    tiles = ((tokens + 127) / 128) * ((features + 63) / 64);
  } else {
    tiles = ((tokens + 127) / 128) * ((features + 255) / 256);
  }
  if (tiles >= 96 || kb < 8 || tokens > 512)
    return pg_gemm_bf16(x, ldx, w, ldw, h, ldh, bias, h, ldh, tokens, features, K, PG_EPI_F32, 0, scale, swap, 1, stream);
  int split = (swap ? 2 * sms : sms) / tiles;
  if (split > kb / 4) split = kb / 4;
  return pg_gemm_bf16(x, ldx, w, ldw, h, ldh, bias, nullptr, 0, tokens, features, K, PG_EPI_ATOMIC_F32, 0, scale, swap, split < 1 ? 1 : split, stream);
}

static int linear_f32(const void* x, long long ldx, const void* w, long long ldw, float* out, long long ldo, int tokens, int features, int K, bool zeros, void* stream) {
  if (tokens <= 0 || features <= 0 || K <= 0 || out == nullptr) return PG_ERR_ARG;
  const int tiles = (features + 127) / 128, kb = (K + 63) / 64, swap = tokens <= 128 ? 1 : 0;
  int split = 2 * pg::num_sms() / tiles;
  if (split > kb / 4) split = kb / 4;
  if (!swap || split <= 1 || pg_gemm_sums_once(tokens, features, K, out, ldo, nullptr, swap))
    return pg_gemm_bf16(x, ldx, w, ldw, out, ldo, nullptr, nullptr, 0, tokens, features, K, PG_EPI_F32, 0, 1.f, swap, 1, stream);
  // few tiles of a long K: split-K partials are red.add-ed into the zeroed output (one row has no pitch: any ldo goes with it)
  const size_t row = features * sizeof(float);
  if (!zeros && cudaMemset2DAsync(out, tokens == 1 ? row : ldo * sizeof(float), 0, row, tokens, reinterpret_cast<cudaStream_t>(stream)) != cudaSuccess) {
    cudaGetLastError();  // do not leave a sticky error behind
    return PG_ERR_CUDA;
  }
  return pg_gemm_bf16(x, ldx, w, ldw, out, ldo, nullptr, nullptr, 0, tokens, features, K, PG_EPI_ATOMIC_F32, 0, 1.f, swap, split, stream);
}

extern "C" int pg_linear_f32(const void* x, long long ldx, const void* w, long long ldw, float* out, long long ldo, int tokens, int features, int K,
                             void* stream) {
  return linear_f32(x, ldx, w, ldw, out, ldo, tokens, features, K, false, stream);
}

extern "C" int pg_linear_f32_zeros(const void* x, long long ldx, const void* w, long long ldw, float* out, long long ldo, int tokens, int features, int K,
                                   void* stream) {
  return linear_f32(x, ldx, w, ldw, out, ldo, tokens, features, K, true, stream);
}

#define PG_TRY(call)                  \
  do {                                \
    const int rc_ = (call);           \
    if (rc_ != PG_OK) return rc_;     \
  } while (0)

extern "C" int pg_siglip_layers(const PgSiglipLayer* layers, int count, float* x, void* hn, void* qkv, void* att, void* mid, int images, int patches,
                                int D, int F, int heads, float eps, void* stream) {
  if (layers == nullptr || count < 0 || images <= 0 || patches <= 0 || heads <= 0 || D <= 0 || D % heads != 0) return PG_ERR_ARG;
  const pg::WeightsFollow chain;
  const int M = images * patches, dh = D / heads;
  const long long N = patches, D3 = 3LL * D;
  const char* q = static_cast<const char*>(qkv);
  for (int i = 0; i < count; ++i) {
    const PgSiglipLayer& l = layers[i];
    PG_TRY(pg_layernorm(x, l.ln1_w, l.ln1_b, hn, nullptr, M, D, eps, stream));
    PG_TRY(pg_gemm_bf16(hn, D, l.qkv_w, D, qkv, D3, l.qkv_b, nullptr, 0, M, 3 * D, D, PG_EPI_BF16, 0, 1.f, 0, 1, stream));
    PG_TRY(pg_attention_prefill(q, q + 2LL * D, q + 4LL * D, att, images, heads, patches, patches, dh, 1, N * D3, D3, 0, dh, N * D3, D3, dh, N * D, D, 0,
                                dh, static_cast<float>(1.0 / std::sqrt(static_cast<double>(dh))), stream));
    PG_TRY(pg_gemm_residual(att, D, l.out_w, D, x, D, l.out_b, M, D, D, 1.f, stream));
    PG_TRY(pg_layernorm(x, l.ln2_w, l.ln2_b, hn, nullptr, M, D, eps, stream));
    PG_TRY(pg_gemm_bf16(hn, D, l.fc1_w, D, mid, F, l.fc1_b, nullptr, 0, M, F, D, PG_EPI_BF16, 1, 1.f, 0, 1, stream));
    PG_TRY(pg_gemm_residual(mid, F, l.fc2_w, F, x, D, l.fc2_b, M, D, F, 1.f, stream));
  }
  return PG_OK;
}

extern "C" int pg_gemma_prefill_layers(const PgGemmaLayer* layers, int count, const PgGemmaPrefill* a, void* stream) {
  if (layers == nullptr || a == nullptr || count < 0 || a->B <= 0 || a->S <= 0 || a->Hkv <= 0 || a->Hq % a->Hkv != 0) return PG_ERR_ARG;
  const pg::WeightsFollow chain;
  const int T = a->B * a->S, D = a->D, F = a->F, Hq = a->Hq, Hkv = a->Hkv, dh = a->dh, G = Hq / Hkv, swap = T > 128 ? 0 : 1;
  const long long W = (Hq + 2LL * Hkv) * dh, S = a->S, qs = a->fused ? W : (long long)Hq * dh, kvs = a->fused ? W : (long long)Hkv * dh, os = (long long)Hq * dh;
  const char* qkv = static_cast<const char*>(a->qkv);
  const void* q = a->fused ? qkv : a->q;
  const void* k = a->fused ? qkv + 2LL * Hq * dh : a->k;
  const void* v = a->fused ? qkv + 2LL * (Hq + Hkv) * dh : a->v;
  const float scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(dh)));
  for (int i = 0; i < count; ++i) {
    const PgGemmaLayer& l = layers[i];
    void* kp = a->k_pages == nullptr ? nullptr : static_cast<char*>(a->k_pages) + i * a->layer_bytes;
    void* vp = a->v_pages == nullptr ? nullptr : static_cast<char*>(a->v_pages) + i * a->layer_bytes;
    PG_TRY(pg_rmsnorm(a->h, l.ln1, a->hn, T, D, a->eps, stream));
    if (a->fused) {
      PG_TRY(pg_gemm_qkv_rope(a->hn, D, l.qkv_w, D, a->qkv, W, T, D, Hq, Hkv, dh, a->pos, a->inv_freq, kp, vp, a->page_table, a->slot_base, a->S, a->page,
                              a->max_pages, stream));
    } else {
      PG_TRY(pg_gemm_bf16(a->hn, D, l.qkv_w, D, a->qkv, W, nullptr, nullptr, 0, T, static_cast<int>(W), D, PG_EPI_BF16, 0, 1.f, swap, 1, stream));
      PG_TRY(pg_rope_kv_append(a->qkv, 0, a->pos, a->q, a->k, a->v, kp, vp, a->page_table, a->slot_base, a->B, a->S, Hq, Hkv, dh, a->page, a->max_pages,
                               a->inv_freq, stream));
    }
    // the G query heads of a k/v head are consecutive rows of one attention problem
    if (a->lens == nullptr)
      PG_TRY(pg_attention_prefill(q, k, v, a->att, a->B, Hkv, a->S * G, a->S, dh, G, S * qs, qs, dh, (long long)G * dh, S * kvs, kvs, dh, S * os, os, dh,
                                  (long long)G * dh, scale, stream));
    else
      PG_TRY(pg_attention_prefill_varlen(q, k, v, a->att, a->lens, a->B, Hkv, a->S * G, a->S, dh, G, S * qs, qs, dh, (long long)G * dh, S * kvs, kvs, dh, S * os,
                                         os, dh, (long long)G * dh, scale, stream));
    PG_TRY(pg_gemm_residual(a->att, os, l.o_w, os, a->h, D, nullptr, T, D, static_cast<int>(os), 1.f, stream));
    PG_TRY(pg_rmsnorm(a->h, l.ln2, a->hn, T, D, a->eps, stream));
    PG_TRY(pg_gemm_bf16(a->hn, D, l.gu_w, D, a->mid, F, nullptr, nullptr, 0, T, 2 * F, D, PG_EPI_GEGLU, 0, 1.f, swap, 1, stream));
    PG_TRY(pg_gemm_residual(a->mid, F, l.down_w, F, a->h, D, nullptr, T, D, F, 1.f, stream));
  }
  return PG_OK;
}

namespace {
// Pieces of one scratch buffer, each on a 256-byte boundary; with no base only their sizes are counted.
struct Pieces {
  char* base;
  long long used = 0;
  explicit Pieces(void* b) : base(static_cast<char*>(b)) {}
  template <typename T>
  T* take(long long n) {
    T* p = base == nullptr ? nullptr : reinterpret_cast<T*>(base + used);
    used += (n * static_cast<long long>(sizeof(T)) + 255) / 256 * 256;
    return p;
  }
};
struct RoutedScratch {
  float *z, *wts, *eo, *shared;
  int *ids, *counts, *offsets, *fill, *plan, *sorted_pair, *pair_row;
  uint16_t *xg, *mid, *smid;
  int pairs, max_tiles;
  long long bytes;
};
RoutedScratch routed_scratch(const PgRoutedFf& a, void* base) {
  RoutedScratch s;
  Pieces p(base);
  s.pairs = a.tokens * a.top;
  s.max_tiles = (s.pairs + pg_moe_tile_rows() - 1) / pg_moe_tile_rows() + a.n_real;
  s.z = p.take<float>(static_cast<long long>(a.tokens) * a.n_pad);
  s.ids = p.take<int>(s.pairs);
  s.wts = p.take<float>(s.pairs);
  s.counts = p.take<int>(a.n_real);
  s.offsets = p.take<int>(a.n_real + 1);
  s.fill = p.take<int>(a.n_real);
  s.plan = p.take<int>(4 + 3LL * s.max_tiles);
  s.sorted_pair = p.take<int>(s.pairs);
  s.pair_row = p.take<int>(s.pairs);
  s.xg = p.take<uint16_t>(static_cast<long long>(s.pairs) * a.D);
  s.mid = p.take<uint16_t>(static_cast<long long>(s.pairs) * a.F);
  s.eo = p.take<float>(static_cast<long long>(s.pairs) * a.D);
  s.smid = p.take<uint16_t>(a.shared_up != nullptr ? static_cast<long long>(a.tokens) * a.shared_F : 0);
  s.shared = p.take<float>(a.shared_up != nullptr ? static_cast<long long>(a.tokens) * a.D : 0);
  s.bytes = p.used;
  return s;
}
}  // namespace

extern "C" long long pg_routed_ff_scratch(const PgRoutedFf* a) {
  if (a == nullptr || a->tokens <= 0 || a->top <= 0 || a->n_real <= 0 || a->D <= 0 || a->F <= 0) return 0;
  return routed_scratch(*a, nullptr).bytes;
}

// The launches of RoutedFeedForward for a step of few rows, issued by one call: eleven from Python cost 150 us of host time, more than the kernels of 300 tokens
// take (109 -> 90 us for top 4 of 14 experts 2048 x 1024 with a shared one of 2048).  Same launches, same order, but for few pairs the plan in one.
extern "C" int pg_routed_ff(const PgRoutedFf* args, const void* h, long long ldh, float* y, int accumulate, void* scratch, long long scratch_bytes, void* stream) {
  if (args == nullptr || h == nullptr || y == nullptr || scratch == nullptr || pg_routed_ff_scratch(args) == 0 || (reinterpret_cast<uintptr_t>(scratch) & 255) != 0) return PG_ERR_ARG;
  const PgRoutedFf& a = *args;
  const RoutedScratch s = routed_scratch(a, scratch);
  if (scratch_bytes < s.bytes || s.max_tiles > 65535) return PG_ERR_ARG;
  const int T = a.tokens;
  PG_TRY(pg_linear_f32(h, ldh, a.router, a.D, s.z, a.n_pad, T, a.n_pad, a.D, stream));
  if (s.pairs <= 4096 && a.n_real <= 1024) {  // (what one CTA plans)
    PG_TRY(pg_moe_route_plan(s.z, a.n_pad, a.correction, s.ids, s.wts, s.offsets, s.plan, s.sorted_pair, s.pair_row, T, a.n_all, a.n_real, a.top, a.group_count, a.group_keep, a.scale,
                             a.router_b, a.flags, s.max_tiles, stream));
  } else {
    PG_TRY(pg_moe_route(s.z, a.n_pad, a.correction, s.ids, s.wts, s.counts, T, a.n_all, a.n_real, a.top, a.group_count, a.group_keep, a.scale, a.router_b, a.flags, stream));
    PG_TRY(pg_moe_plan(s.counts, s.ids, s.offsets, s.fill, s.plan, s.sorted_pair, s.pair_row, s.pairs, a.n_real, s.max_tiles, stream));
  }
  PG_TRY(pg_moe_products(h, ldh, s.sorted_pair, s.offsets + a.n_real, a.top, s.xg, a.w_up, a.w_down, s.mid, s.eo, s.plan, s.max_tiles, s.pairs, a.n_real, a.D, a.F, a.act,
                         stream));
  if (a.shared_up != nullptr) {
    PG_TRY(pg_gemm_bf16(h, ldh, a.shared_up, a.D, s.smid, a.shared_F, nullptr, nullptr, 0, T, a.shared_F, a.D, PG_EPI_BF16, 2, 1.f, T <= 128 ? 1 : 0, 1, stream));
    PG_TRY(pg_linear_f32(s.smid, a.shared_F, a.shared_down, a.shared_F, s.shared, a.D, T, a.D, a.shared_F, stream));
  }
  return pg_moe_combine(s.eo, a.D, s.pair_row, s.ids, s.wts, h, ldh, a.shared_up != nullptr ? s.shared : nullptr, a.D, y, T, a.D, a.top, 0,
                        a.shared_gate ? s.z + a.n_all : nullptr, a.n_pad, accumulate, stream);
}
