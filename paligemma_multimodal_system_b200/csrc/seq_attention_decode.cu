// Attention of single new tokens (decode rows: entries with one new token) over the paged cache, rows of whole 16-byte pieces: heads of a multiple of
// eight elements, values up to 128 wide, pages of a multiple of 32 keys.  (Other rows: attn_decode_kernel in seq_mixers.cu.)
//
// CTA = (key split, k/v head, entry), four warps; a warp walks 32-key tiles of its own straight from the pages, no block-wide barrier in the loop.  What bounds
// it: the bytes of the keys and values where there are many, else a chain of round trips (descriptors, page, keys, merge).  So
//   * eight lanes share a key row (16 bytes each, eight keys a lane), a load instruction covers whole 128-byte lines of four keys, and the 32 partial dot
//     products of a lane (8 keys x 4 heads) are summed over the eight lanes by halving exchanges: 28 shuffles, after which a lane holds the scores of one key;
//   * the values of the tile are requested before the scores are summed and exponentiated (64-wide bf16 heads);
//   * probabilities are exchanged as one float4 per key (four heads), the row sums stay per lane until the end;
//   * 128 threads of up to 168 registers leave three CTAs on an SM: 48 requests x 8 k/v heads are one wave.
// One query head group of four per pass; larger groups walk the keys again.
// 48 requests x 8 k/v heads x 64, ~240 keys, in their step: 33 -> 19 us.  Whole sub-layers of 2048: 64 requests x ~2250 keys 240 -> 172 us, 40 x ~820 78 -> 59,
// one x 3000 50 -> 41; fp32 64 x ~2250 336 -> 244, 24 x ~375 65 -> 59.
#include "common.cuh"
#include "paligemma_b200.h"

using bf16 = __nv_bfloat16;

namespace {

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float wmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float sigmoidf(float z) { return 1.0f / (1.0f + expf(-z)); }

template <typename T>
struct Row8;  // eight neighbouring elements as they lie in memory
template <>
struct Row8<bf16> {
  uint4 u;
  __device__ __forceinline__ void load(const bf16* p) { u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void zero() { u = make_uint4(0, 0, 0, 0); }
  __device__ __forceinline__ void get(float (&v)[8]) const {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};
template <>
struct Row8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) { a = reinterpret_cast<const float4*>(p)[0]; b = reinterpret_cast<const float4*>(p)[1]; }
  __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void get(float (&v)[8]) const {
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
};
__device__ __forceinline__ float ldf(const float* p, long long i) { return p[i]; }
__device__ __forceinline__ float ldf(const bf16* p, long long i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void stf(float* p, long long i, float v) { p[i] = v; }
__device__ __forceinline__ void stf(bf16* p, long long i, float v) { p[i] = __float2bfloat16_rn(v); }

constexpr int kWarps = 4;

// VC = ceil(vdim / 64): 64-column pieces of a value row.  LOGI: weights sigmoid(score + bias), unnormalised.
template <typename TA, int VC, bool LOGI>
__global__ void __launch_bounds__(32 * kWarps, VC == 1 && sizeof(TA) == 2 ? 3 : 2) attn_decode_vec_kernel(const TA* __restrict__ q, const TA* __restrict__ k_pages, const TA* __restrict__ v_pages,
                                                                         const TA* __restrict__ gate, long long ldg, TA* __restrict__ out, float* __restrict__ partial,
                                                                         const int* __restrict__ entry_row0, const int* __restrict__ entry_n,
                                                                         const int* __restrict__ entry_ctx, const int* __restrict__ page_table, int max_pages,
                                                                         int page, int H, int G, int dim, int vdim, float scale, float softcap, long long krow,
                                                                         long long vrow, int gate_per_head, PgAttnScore sx, int trigger) {
  constexpr bool EARLY_V = VC == 1 && sizeof(TA) == 2;
  const int e = blockIdx.z, g = blockIdx.y, split = blockIdx.x, nsplit = gridDim.x, gsz = H / G;
  const int ctx = entry_ctx[e];
  const long long t = entry_row0[e];
  const bool mine = entry_n[e] == 1;
  const int chunks = (dim + 63) / 64, dimp = 64 * chunks;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                          // [gsz][dimp], zeros past dim
  float4* Pw = reinterpret_cast<float4*>(Qs + gsz * dimp);   // [kWarps][32] the four heads' weights of a key
  float* Mg = reinterpret_cast<float*>(Pw + kWarps * 32);    // [kWarps][4] max, [kWarps][4] sum, then [kWarps][4][vdim] accumulators
  float* Lg = Mg + kWarps * 4;
  float* Og = Lg + kWarps * 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kg = lane >> 3, l8 = lane & 7;
  const long long ldo = sx.out_ld > 0 ? sx.out_ld : (long long)H * vdim;
  const float oscale = sx.out_scale != 0.f ? sx.out_scale : 1.f;
  const int* pt = page_table + (long long)e * max_pages;
  const int ntiles = ctx / 32 + 1;  // keys 0 .. ctx
  // with a window only the tiles of the kept first keys [0, nk) and of the window [t_lo, ntiles) are walked
  const int window = sx.window > 0 ? sx.window : 0x3fffffff, keep = sx.window > 0 ? max(sx.keep_first, 0) : 0;
  const int t_lo = max(0, ctx - window + 1) / 32;
  const int nkeep = min(min((keep + 31) / 32, ntiles), t_lo);
  const int nwalk = nkeep + ntiles - t_lo;
  // the keys and values of earlier steps, on their way to L2 while the kernels before still run (only a hint: whatever those write is read behind the wait)
  if (mine)
    for (int w = 0, walk = split * kWarps + warp; w < 4 && walk < nwalk; ++w, walk += nsplit * kWarps) {
      const int it = walk < nkeep ? walk : t_lo + (walk - nkeep);
      const long long row = (long long)pt[(it * 32) / page] * page + (it * 32) % page + lane;
      const char* k = reinterpret_cast<const char*>(k_pages + row * krow + (long long)g * dim);
      const char* v = reinterpret_cast<const char*>(v_pages + row * vrow + (long long)g * vdim);
      for (int i = 0; i < dim * (int)sizeof(TA); i += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(k + i));
      for (int i = 0; i < vdim * (int)sizeof(TA); i += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(v + i));
    }
  pg::griddep_begin_if(trigger);
  if (!mine) return;
  for (int i = threadIdx.x; i < gsz * dimp; i += 32 * kWarps) {
    const int r = i / dimp, d = i % dimp;
    Qs[i] = d < dim ? ldf(q, t * ((long long)H * dim) + (long long)(g * gsz + r) * dim + d) : 0.f;
  }
  __syncthreads();
  for (int rb = 0; rb < gsz; rb += 4) {
    const int nr = min(4, gsz - rb);
    float m[4], l[4], o[4][8 * VC];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = LOGI ? 0.f : -INFINITY; l[i] = 0.f;  // LOGI: a constant maximum, so that partial sums merge with factor one
#pragma unroll
      for (int c = 0; c < 8 * VC; ++c) o[i][c] = 0.f;
    }
    for (int walk = split * kWarps + warp; walk < nwalk; walk += nsplit * kWarps) {
      const int it = walk < nkeep ? walk : t_lo + (walk - nkeep);
      const long long row0 = (long long)pt[(it * 32) / page] * page + (it * 32) % page;  // (a tile never straddles a page)
      const TA* kt = k_pages + (row0 + kg) * krow + (long long)g * dim + 8 * l8;
      const TA* vt = v_pages + (row0 + kg) * vrow + (long long)g * vdim + 8 * l8;
      Row8<TA> vv[EARLY_V ? 8 : 1];
      float s[8][4];
#pragma unroll
      for (int x = 0; x < 8; ++x)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[x][i] = 0.f;
      for (int c = 0; c < chunks; ++c) {
        if (64 * c + 8 * l8 < dim) {
          float qv[4][8];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4* qp = reinterpret_cast<const float4*>(Qs + min(rb + i, gsz - 1) * dimp + 64 * c + 8 * l8);
            const float4 a = qp[0], b = qp[1];
            qv[i][0] = a.x; qv[i][1] = a.y; qv[i][2] = a.z; qv[i][3] = a.w; qv[i][4] = b.x; qv[i][5] = b.y; qv[i][6] = b.z; qv[i][7] = b.w;
          }
          Row8<TA> kk[8];
#pragma unroll
          for (int x = 0; x < 8; ++x) kk[x].load(kt + (long long)(4 * x) * krow + 64 * c);  // (rows past ctx lie in the same page; their scores are masked)
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            float kv[8];
            kk[x].get(kv);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int d = 0; d < 8; ++d) s[x][i] = fmaf(qv[i][d], kv[d], s[x][i]);
          }
        }
      }
      if (EARLY_V) {
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          if (it * 32 + 4 * x + kg <= ctx && 8 * l8 < vdim) vv[EARLY_V ? x : 0].load(vt + (long long)(4 * x) * vrow);
          else vv[EARLY_V ? x : 0].zero();
        }
      }
      // sums over the eight lanes of a row; lane (kg, l8) ends with the scores of key 4 l8 + kg
#pragma unroll
      for (int w = 4; w >= 1; w >>= 1) {
        const bool up = (l8 & w) != 0;
#pragma unroll
        for (int x = 0; x < w; ++x)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float mine = up ? s[x + w][i] : s[x][i], theirs = up ? s[x][i] : s[x + w][i];
            s[x][i] = mine + __shfl_xor_sync(0xffffffffu, theirs, w);
          }
      }
      const int j = it * 32 + 4 * l8 + kg;
      const bool vis = j <= ctx && (ctx - j < window || j < keep);
      float pr[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int head = g * gsz + min(rb + i, gsz - 1);
        float sc = s[0][i] * (scale * (sx.head_scale != nullptr ? sx.head_scale[head] : 1.f));
        if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
        if (sx.dist_a != nullptr && vis) sc -= sx.dist_a[head] * log1pf(sx.dist_b[head] * (float)(ctx - j));
        sc = vis ? sc : -INFINITY;
        if (LOGI) {
          pr[i] = vis ? sigmoidf(sc + (sx.head_bias != nullptr ? sx.head_bias[head] : 0.f)) : 0.f;
        } else {
          const float mn = fmaxf(m[i], wmax(sc));  // every walked tile holds a visible key: mn is finite
          pr[i] = vis ? expf(sc - mn) : 0.f;
          const float corr = expf(m[i] - mn);
          l[i] = l[i] * corr + pr[i];
          m[i] = mn;
#pragma unroll
          for (int c = 0; c < 8 * VC; ++c) o[i][c] *= corr;
        }
      }
      float4* pw = Pw + warp * 32;
      pw[4 * l8 + kg] = make_float4(pr[0], pr[1], pr[2], pr[3]);
      __syncwarp();
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        if (EARLY_V || 64 * c + 8 * l8 < vdim) {
          Row8<TA> ww[EARLY_V ? 1 : 8];
          if (!EARLY_V) {
#pragma unroll
            for (int x = 0; x < 8; ++x) {
              if (it * 32 + 4 * x + kg <= ctx) ww[EARLY_V ? 0 : x].load(vt + (long long)(4 * x) * vrow + 64 * c);
              else ww[EARLY_V ? 0 : x].zero();
            }
          }
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            float v[8];
            if (EARLY_V) vv[EARLY_V ? x : 0].get(v);
            else ww[EARLY_V ? 0 : x].get(v);
            const float4 p = pw[4 * x + kg];
#pragma unroll
            for (int d = 0; d < 8; ++d) {
              o[0][8 * c + d] = fmaf(p.x, v[d], o[0][8 * c + d]);
              o[1][8 * c + d] = fmaf(p.y, v[d], o[1][8 * c + d]);
              o[2][8 * c + d] = fmaf(p.z, v[d], o[2][8 * c + d]);
              o[3][8 * c + d] = fmaf(p.w, v[d], o[3][8 * c + d]);
            }
          }
        }
      }
      __syncwarp();
    }
    // the four key groups of the warp, then the warps
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int c = 0; c < 8 * VC; ++c) {
        o[i][c] += __shfl_xor_sync(0xffffffffu, o[i][c], 8);
        o[i][c] += __shfl_xor_sync(0xffffffffu, o[i][c], 16);
      }
      l[i] = wsum(l[i]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (lane == 0) { Mg[warp * 4 + i] = m[i]; Lg[warp * 4 + i] = l[i]; }
      if (kg == i) {
#pragma unroll
        for (int c = 0; c < VC; ++c)
          if (64 * c + 8 * l8 < vdim) {
            float4* dst = reinterpret_cast<float4*>(Og + (warp * 4 + i) * vdim + 64 * c + 8 * l8);
            dst[0] = make_float4(o[i][8 * c], o[i][8 * c + 1], o[i][8 * c + 2], o[i][8 * c + 3]);
            dst[1] = make_float4(o[i][8 * c + 4], o[i][8 * c + 5], o[i][8 * c + 6], o[i][8 * c + 7]);
          }
      }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nr * vdim; idx += 32 * kWarps) {
      const int i = idx / vdim, col = idx % vdim;
      const int head = g * gsz + rb + i;
      float gt = 0.f;
      if (nsplit == 1 && gate != nullptr) gt = ldf(gate, t * ldg + (gate_per_head ? (long long)head : (long long)head * vdim + col));
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) M = fmaxf(M, Mg[w * 4 + i]);
      float acc = 0.f, ls = 0.f;
      if (M > -INFINITY) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          const float f = expf(Mg[w * 4 + i] - M);
          acc = fmaf(f, Og[(w * 4 + i) * vdim + col], acc);
          ls = fmaf(f, Lg[w * 4 + i], ls);
        }
      }
      if (nsplit == 1) {
        if (!LOGI && sx.sink != nullptr) {
          const float sk = sx.sink[head], mm = fmaxf(M, sk), f = expf(M - mm);
          acc *= f;
          ls = ls * f + expf(sk - mm);
        }
        float v = (LOGI ? acc : acc / ls) * oscale;
        if (gate != nullptr) v *= sigmoidf(gt);
        stf(out, t * ldo + (long long)head * vdim + col, v);
      } else {
        float* pp = partial + (((long long)e * H + head) * nsplit + split) * (vdim + 2);
        pp[2 + col] = acc;
        if (col == 0) { pp[0] = M; pp[1] = ls; }
      }
    }
  }
}

template <typename TA, int VC>
int launch(const void* q, const void* kp, const void* vp, const void* gate, long long ldg, void* out, float* partial, const int* row0, const int* n,
           const int* ctx, const int* pt, int max_pages, int page, int entries, int nsplit, int H, int G, int dim, int vdim, float scale, float softcap,
           long long krow, long long vrow, int gate_per_head, const PgAttnScore& sx, cudaStream_t st) {
  const int gsz = H / G, dimp = (dim + 63) / 64 * 64;
  const size_t smem = ((size_t)gsz * dimp + kWarps * (128 + 8 + (size_t)4 * vdim)) * sizeof(float);
  constexpr int kMost = 200 * 1024;
  if (smem > kMost) return PG_ERR_ARG;
  auto kern = sx.logistic ? attn_decode_vec_kernel<TA, VC, true> : attn_decode_vec_kernel<TA, VC, false>;
  // once a device, to the most that any call asks for: calls of several threads find the same
  static bool configured[2][pg::kMaxDevices] = {};
  bool& done = configured[sx.logistic ? 1 : 0][pg::current_device()];
  if (!done) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost) != cudaSuccess) {
      cudaGetLastError();
      return PG_ERR_CUDA;
    }
    done = true;
  }
  return pg::launch_kernel(kern, dim3(nsplit, G, entries), dim3(32 * kWarps), smem, st, static_cast<const TA*>(q), static_cast<const TA*>(kp),
                           static_cast<const TA*>(vp), static_cast<const TA*>(gate), ldg, static_cast<TA*>(out), partial, row0, n, ctx, pt, max_pages, page, H, G,
                           dim, vdim, scale, softcap, krow, vrow, gate_per_head, sx, pg::weights_follow()) == cudaSuccess
             ? PG_OK : PG_ERR_CUDA;
}

}  // namespace

int pg_attn_decode_vec(const void* q, const void* kp, const void* vp, const void* gate, long long ldg, void* out, float* partial, const int* row0,
                       const int* n, const int* ctx, const int* pt, int max_pages, int page, int entries, int nsplit, int H, int G, int dim, int vdim,
                       float scale, float softcap, int act_f32, long long krow, long long vrow, int gate_per_head, const PgAttnScore& sx, cudaStream_t st) {
#define PG_DV(TA, VC) \
  return launch<TA, VC>(q, kp, vp, gate, ldg, out, partial, row0, n, ctx, pt, max_pages, page, entries, nsplit, H, G, dim, vdim, scale, softcap, krow, vrow, gate_per_head, sx, st)
  if (act_f32) {
    if (vdim <= 64) PG_DV(float, 1);
    PG_DV(float, 2);
  }
  if (vdim <= 64) PG_DV(bf16, 1);
  PG_DV(bf16, 2);
#undef PG_DV
}
