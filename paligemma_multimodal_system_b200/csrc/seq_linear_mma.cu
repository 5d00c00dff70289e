// Decayed linear attention of prompt portions in bf16 on the tensor cores (the block form of pg_linear_attn_scan),
// with every quantity of the recurrence at fp32 precision: queries and keys are turned and scaled (or, with SILU, queries, keys and values activated) in fp32 as they are staged and enter
// the products as three bf16 terms (8 + 8 + 8 mantissa bits), as do the state and the decay-weighted scores and values.
//
// With a = decay, block rows i, j = 0 .. c-1 and S the state before the block:
//   o_i = a^(i+1) S^T q_i + sum_{j <= i} P_ij v_j,  P_ij = a^(i-j) (q_i . k_j);      S' = a^c S + sum_j a^(c-1-j) k_j v_j^T
//
// A CTA advances 64 value columns of one head of one entry through all its new tokens.  The state is held TRANSPOSED, S^T [value column, key
// dimension], as the fp32 accumulators of m16n8k16 tiles (warp = 16 value columns): two adjacent 8-column accumulator tiles are, element
// for element, the A operand of a 16-deep product step.  The tensor pipe cuts its sums off where fp32 would round, always towards zero, so few products meet a sum of
// full size: the leading ones (first term by first term) have accumulators of their own, over at most four steps, the others gather apart, and whole sums are added and
// rounded in fp32 (all products of a block on one accumulator: 1.3e-6 against 64 bits where it is 7.9e-8 now).  The raw rows of the next block and its cosines / sines are fetched into registers,
// its values with cp.async (SILU: into registers as well; they are staged as three terms), while the current block is multiplied.
//
// What bounds it: the mma.sync pipe, six products for one of fp32, and between them the cuts into terms; two CTAs per SM, or three (see the dispatch).  Blocks are 32 tokens: with 64 the
// accumulators of their own do not fit the registers (without silu, 48 prompts of 193 .. 256 tokens, 16 heads, blocks of 64 / 32: 64 wide 126 / 97 us, 32 wide 72 / 62; 2 x 1000 tokens 118 /
// 81; 64 with one accumulator, six times the error: 107, 69, 90).
// SILU, 48 prompts of 193 .. 256 tokens, 32 heads of 64: FMA chains over blocks of 32 (linear_attn_chunked_kernel, bound by its shared-memory operands) 570 us, here 283; the error
// against 64 bits 1.6e-7 there, 0.8e-7 here.
#include "common.cuh"
#include "paligemma_b200.h"

using bf16 = __nv_bfloat16;
using pg::cp_async16;
using pg::ldmatrix_x4;
using pg::ldmatrix_x4_trans;
using pg::mma_bf16_16816;
using pg::smem_u32;

namespace {

__device__ __forceinline__ float lo_f(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi_f(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// (p, q) = sum of three bf16 pairs, packed
__device__ __forceinline__ void cut3(float p, float q, uint32_t& a, uint32_t& b, uint32_t& c) {
  a = pg::pack_bf16(p, q);
  const float p1 = p - lo_f(a), q1 = q - hi_f(a);
  b = pg::pack_bf16(p1, q1);
  c = pg::pack_bf16(p1 - lo_f(b), q1 - hi_f(b));
}

// as linear_attn_chunked_kernel: bf16 projections carry 8 mantissa bits, so their silu may use the hardware exponential and reciprocal
__device__ __forceinline__ float silu_of_bf16(float z) { return z * __frcp_rn(1.0f + __expf(-z)); }

template <int DIM, int C, bool SILU, int CTAS>
__global__ void __launch_bounds__(128, CTAS) linear_attn_block_kernel(const bf16* __restrict__ qkv, long long ld, float* __restrict__ state,
                                                                   const float* __restrict__ decay, float* __restrict__ out,
                                                                   const int* __restrict__ entry_row0, const int* __restrict__ entry_n,
                                                                   const int* __restrict__ entry_ctx, const int* __restrict__ entry_slot, int H, int dim,
                                                                   int vdim, PgLinearAttnOps ops) {
  pg::griddep_begin();
  constexpr int LD = DIM + 8, LV = 64 + 8, LP = C + 8, CH = DIM / 8, NI = C * CH / 128, TILE = C * LD, R = C / 16;
  // leading products apart (see above): not for the wide heads of layers without silu, whose registers do not hold them (128 wide, 4 x 300 tokens, 16 heads: 60 us, apart 72)
  constexpr bool APART = SILU || DIM <= 64;
  constexpr int PAR = DIM <= 64 ? 2 : 1;  // accumulators of the leading products with the state
  constexpr int VT = SILU ? 3 : 1, NV = SILU ? C * 8 / 128 : 1;  // terms of a value; pieces of the values that a thread stages
  static_assert(C * CH % 128 == 0, "every thread stages the same number of 8-element pieces");
  const int e = blockIdx.z, h = blockIdx.y;
  const int n = entry_n[e];
  if (n < ops.n_min || n > ops.n_max) return;
  const long long row0 = entry_row0[e];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  extern __shared__ __align__(16) unsigned char smraw[];
  bf16* Qs = reinterpret_cast<bf16*>(smraw);  // [3 terms][C][LD]
  bf16* Ks = Qs + 3 * TILE;                   // [3 terms][C][LD]
  bf16* Ps = Ks + 3 * TILE;                   // [3 terms][C][LP]
  bf16* Vs = Ps + 3 * C * LP;                 // [2 buffers][C][LV]; SILU: [3 terms][C][LV]
  float* ap = reinterpret_cast<float*>(Vs + (SILU ? 3 : 2) * C * LV);  // a^0 .. a^C
  const int v_base = blockIdx.x * 64, vcol = v_base + warp * 16 + gq;
  const bf16* qp = qkv + (long long)h * dim;
  const bf16* kp = qkv + (long long)(H + h) * dim;
  const bf16* vp = qkv + 2LL * H * dim + (long long)h * vdim + v_base;
  float* stp = state + (((long long)entry_slot[e] * H + h) * dim) * vdim;
  const bool fresh = entry_ctx[e] == 0;
  float S[DIM / 8][4];
#pragma unroll
  for (int nb = 0; nb < DIM / 8; ++nb)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = nb * 8 + 2 * tq + (i & 1), c = vcol + (i >> 1) * 8;
      S[nb][i] = (!fresh && d < dim && c < vdim) ? stp[(long long)d * vdim + c] : 0.f;
    }
  for (int i = tid; i <= C; i += 128) ap[i] = (float)pow((double)decay[h], (double)i);
  uint4 rq[NI], rk[NI], rv[NV];
  float4 rc[SILU ? 1 : NI], rs[SILU ? 1 : NI];
  auto fetch = [&](int t0, int buf) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int id = tid + 128 * i, r = id / CH, c = (id % CH) * 8;
      const bool ok = t0 + r < n && c < dim;
      const long long row = row0 + t0 + r;
      rq[i] = ok ? *reinterpret_cast<const uint4*>(qp + row * ld + c) : make_uint4(0, 0, 0, 0);
      rk[i] = ok ? *reinterpret_cast<const uint4*>(kp + row * ld + c) : make_uint4(0, 0, 0, 0);
      if constexpr (SILU) continue;
      const bool turn = ok && ops.rotate != nullptr;
      rc[i] = turn ? *reinterpret_cast<const float4*>(ops.rotate + row * 2 * ops.pairs + c / 2) : make_float4(1.f, 1.f, 1.f, 1.f);
      rs[i] = turn ? *reinterpret_cast<const float4*>(ops.rotate + (row * 2 + 1) * ops.pairs + c / 2) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if constexpr (SILU) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int id = tid + 128 * i, r = id / 8, c = (id % 8) * 8;
        const bool ok = t0 + r < n && v_base + c < vdim;
        rv[i] = ok ? *reinterpret_cast<const uint4*>(vp + (row0 + t0 + r) * ld + c) : make_uint4(0, 0, 0, 0);
      }
      return;
    }
    for (int id = tid; id < C * 8; id += 128) {
      const int r = id / 8, c = (id % 8) * 8;
      const bool ok = t0 + r < n && v_base + c < vdim;
      cp_async16(smem_u32(Vs + (buf * C + r) * LV + c), vp + (row0 + (ok ? t0 + r : 0)) * ld + (ok ? c : 0), ok);
    }
    pg::cp_async_commit();
  };
  auto form_tiles = [&]() {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int id = tid + 128 * i, r = id / CH, c = (id % CH) * 8;
      const uint32_t qw[4] = {rq[i].x, rq[i].y, rq[i].z, rq[i].w}, kw[4] = {rk[i].x, rk[i].y, rk[i].z, rk[i].w};
      const float4 c4 = rc[SILU ? 0 : i], s4 = rs[SILU ? 0 : i];
      const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
      uint32_t t[6][4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float q0 = lo_f(qw[p]), q1 = hi_f(qw[p]), k0 = lo_f(kw[p]), k1 = hi_f(kw[p]);
        if constexpr (SILU) {
          cut3(silu_of_bf16(q0), silu_of_bf16(q1), t[0][p], t[1][p], t[2][p]);
          cut3(silu_of_bf16(k0), silu_of_bf16(k1), t[3][p], t[4][p], t[5][p]);
          continue;
        }
        cut3(q0 * cs[p] - q1 * sn[p], q1 * cs[p] + q0 * sn[p], t[0][p], t[1][p], t[2][p]);
        cut3((k0 * cs[p] - k1 * sn[p]) * ops.kscale, (k1 * cs[p] + k0 * sn[p]) * ops.kscale, t[3][p], t[4][p], t[5][p]);
      }
      bf16* to = Qs + r * LD + c;  // Ks follows Qs: six tiles one after the other
#pragma unroll
      for (int m = 0; m < 6; ++m) *reinterpret_cast<uint4*>(to + m * TILE) = make_uint4(t[m][0], t[m][1], t[m][2], t[m][3]);
    }
    if constexpr (SILU) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int id = tid + 128 * i, r = id / 8, c = (id % 8) * 8;
        const uint32_t vw[4] = {rv[i].x, rv[i].y, rv[i].z, rv[i].w};
        uint32_t t[3][4];
#pragma unroll
        for (int p = 0; p < 4; ++p) cut3(silu_of_bf16(lo_f(vw[p])), silu_of_bf16(hi_f(vw[p])), t[0][p], t[1][p], t[2][p]);
#pragma unroll
        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint4*>(Vs + (m * C + r) * LV + c) = make_uint4(t[m][0], t[m][1], t[m][2], t[m][3]);
      }
    }
  };
  // lane's row / column inside a 16 x 16 block for ldmatrix: A operand (row-major), B operand (rows = n), and their transposed forms
  const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8, a_col = ((lane >> 4) & 1) * 8;
  const int b_row = (lane & 7) + ((lane >> 4) & 1) * 8, b_col = ((lane >> 3) & 1) * 8;
  fetch(0, 0);
  int cur = 0;
  for (int t0 = 0; t0 < n; t0 += C, cur ^= 1) {
    const int cn = min(C, n - t0);
    form_tiles();
    pg::cp_async_wait<0>();
    __syncthreads();  // this block's tiles are there
    if (t0 + C < n) fetch(t0 + C, cur ^ 1);
    const bf16* Vb = SILU ? Vs : Vs + cur * C * LV;
    // P: the 16 x 16 blocks on and below the diagonal, shared out over the warps
    for (int id = warp; id < R * (R + 1) / 2; id += 4) {
      int ib = 0, jb = id;
      while (jb > ib) { jb -= ib + 1; ++ib; }
      float s[2][2][4] = {}, sl[2][2][4] = {};  // leading products and the others, of even and odd steps
#pragma unroll
      for (int kd = 0; kd < DIM / 16; ++kd) {
        uint32_t qa[3][4], kb[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          ldmatrix_x4(smem_u32(Qs + x * TILE + (ib * 16 + a_row) * LD + kd * 16 + a_col), qa[x][0], qa[x][1], qa[x][2], qa[x][3]);
          ldmatrix_x4(smem_u32(Ks + x * TILE + (jb * 16 + b_row) * LD + kd * 16 + b_col), kb[x][0], kb[x][1], kb[x][2], kb[x][3]);
        }
#pragma unroll
        for (int x = 0; x < 6; ++x) {  // two operands in three terms each (dropped products lie below 2^-24)
          constexpr int TERM_A[6] = {0, 0, 1, 1, 0, 2}, TERM_B[6] = {0, 1, 0, 1, 2, 0};
          float(&to)[2][4] = APART ? (x == 0 ? s[kd & 1] : sl[kd & 1]) : s[x & 1];
          mma_bf16_16816(to[0], qa[TERM_A[x]], kb[TERM_B[x]][0], kb[TERM_B[x]][1]);
          mma_bf16_16816(to[1], qa[TERM_A[x]], kb[TERM_B[x]][2], kb[TERM_B[x]][3]);
        }
      }
      const int tl = ib * 16 + gq, th = tl + 8;
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        const int j = jb * 16 + nb * 8 + 2 * tq;
        float p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int away = ((i & 2) ? th : tl) - (j + (i & 1));
          const float sum = APART ? (s[0][nb][i] + s[1][nb][i]) + (sl[0][nb][i] + sl[1][nb][i]) : s[0][nb][i] + s[1][nb][i];
          p[i] = away >= 0 ? sum * ap[away >= 0 ? away : 0] : 0.f;
        }
        uint32_t c[3][2];
        cut3(p[0], p[1], c[0][0], c[1][0], c[2][0]);
        cut3(p[2], p[3], c[0][1], c[1][1], c[2][1]);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          *reinterpret_cast<uint32_t*>(Ps + (x * C + tl) * LP + j) = c[x][0];
          *reinterpret_cast<uint32_t*>(Ps + (x * C + th) * LP + j) = c[x][1];
        }
      }
    }
    // outputs O^T [16 value columns, C tokens]: the part of the carried state (needs no P)
    float o[C / 8][4], ol[C / 8][4];
#pragma unroll
    for (int i = 0; i < C / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    if (!(fresh && t0 == 0)) {
      float oh[PAR][C / 8][4];
#pragma unroll
      for (int i = 0; i < C / 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) ol[i][c] = oh[0][i][c] = oh[PAR - 1][i][c] = 0.f;
#pragma unroll
      for (int kd = 0; kd < DIM / 16; ++kd) {
        uint32_t sa[3][4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          cut3(S[2 * kd + hf][0], S[2 * kd + hf][1], sa[0][2 * hf], sa[1][2 * hf], sa[2][2 * hf]);
          cut3(S[2 * kd + hf][2], S[2 * kd + hf][3], sa[0][2 * hf + 1], sa[1][2 * hf + 1], sa[2][2 * hf + 1]);
        }
#pragma unroll
        for (int y = 0; y < 3; ++y) {
          uint32_t bq[R][4];
#pragma unroll
          for (int tb = 0; tb < R; ++tb)
            ldmatrix_x4(smem_u32(Qs + y * TILE + (tb * 16 + b_row) * LD + kd * 16 + b_col), bq[tb][0], bq[tb][1], bq[tb][2], bq[tb][3]);
#pragma unroll
          for (int x = 0; x < 3 - y; ++x)  // terms (0,0) (1,0) (2,0) (0,1) (1,1) (0,2)
#pragma unroll
            for (int tb = 0; tb < R; ++tb) {
              float(&to)[C / 8][4] = !APART || x + y == 0 ? oh[kd & (PAR - 1)] : ol;
              mma_bf16_16816(to[2 * tb], sa[x], bq[tb][0], bq[tb][1]);
              mma_bf16_16816(to[2 * tb + 1], sa[x], bq[tb][2], bq[tb][3]);
            }
        }
      }
#pragma unroll
      for (int nb = 0; nb < C / 8; ++nb) {
        const float c0 = ap[nb * 8 + 2 * tq + 1], c1 = ap[nb * 8 + 2 * tq + 2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float lead = PAR == 2 ? oh[0][nb][i] + oh[PAR - 1][nb][i] : oh[0][nb][i];
          o[nb][i] = (APART ? lead + ol[nb][i] : lead) * ((i & 1) ? c1 : c0);
        }
      }
    }
    const float carry = ap[cn];
#pragma unroll
    for (int nb = 0; nb < DIM / 8; ++nb) { S[nb][0] *= carry; S[nb][1] *= carry; S[nb][2] *= carry; S[nb][3] *= carry; }
    float oh[C / 8][4];
#pragma unroll
    for (int i = 0; i < C / 8; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) oh[i][c] = ol[i][c] = 0.f;
    float(&sum)[C / 8][4] = APART ? oh : o;
    __syncthreads();  // P is complete
#pragma unroll
    for (int kk = 0; kk < R; ++kk) {
      uint32_t va[VT][4], wa[3][4];
#pragma unroll
      for (int y = 0; y < VT; ++y) ldmatrix_x4_trans(smem_u32(Vb + (y * C + kk * 16 + b_row) * LV + warp * 16 + b_col), va[y][0], va[y][1], va[y][2], va[y][3]);
#pragma unroll
      for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int tb = kk; tb < R; ++tb) {
          uint32_t b0, b1, b2, b3;
          ldmatrix_x4(smem_u32(Ps + (x * C + tb * 16 + b_row) * LP + kk * 16 + b_col), b0, b1, b2, b3);
#pragma unroll
          for (int y = 0; y < (VT < 3 - x ? VT : 3 - x); ++y) {
            float(&to)[C / 8][4] = !APART || x + y == 0 ? sum : ol;
            mma_bf16_16816(to[2 * tb], va[y], b0, b1);
            mma_bf16_16816(to[2 * tb + 1], va[y], b2, b3);
          }
        }
      float v8[8];  // the values (the terms' sums are exact)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v8[2 * i] = lo_f(va[0][i]);
        v8[2 * i + 1] = hi_f(va[0][i]);
        if constexpr (SILU) {
          v8[2 * i] += lo_f(va[VT - 2][i]) + lo_f(va[VT - 1][i]);
          v8[2 * i + 1] += hi_f(va[VT - 2][i]) + hi_f(va[VT - 1][i]);
        }
      }
      // state: values weighted by a^(c-1-j) against the keys
      const int j = kk * 16 + 2 * tq;
      auto weight = [&](int t) { return t < cn ? ap[cn - 1 - t] : 0.f; };
      const float w0 = weight(j), w1 = weight(j + 1), w2 = weight(j + 8), w3 = weight(j + 9);
      cut3(v8[0] * w0, v8[1] * w1, wa[0][0], wa[1][0], wa[2][0]);
      cut3(v8[2] * w0, v8[3] * w1, wa[0][1], wa[1][1], wa[2][1]);
      cut3(v8[4] * w2, v8[5] * w3, wa[0][2], wa[1][2], wa[2][2]);
      cut3(v8[6] * w2, v8[7] * w3, wa[0][3], wa[1][3], wa[2][3]);
#pragma unroll
      for (int dp = 0; dp < DIM / 32; ++dp) {
        float part[4][4] = {};
        auto acc = [&](int i) -> float(&)[4] { return APART ? part[i] : S[4 * dp + i]; };
#pragma unroll
        for (int y = 2; y >= 0; --y) {  // the smallest products first: the leading one is cut off once, the sum joins the state rounded
          uint32_t bk[2][4];
#pragma unroll
          for (int hf = 0; hf < 2; ++hf)
            ldmatrix_x4_trans(smem_u32(Ks + y * TILE + (kk * 16 + a_row) * LD + (2 * dp + hf) * 16 + a_col), bk[hf][0], bk[hf][1], bk[hf][2], bk[hf][3]);
#pragma unroll
          for (int x = 2 - y; x >= 0; --x)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              mma_bf16_16816(acc(2 * hf), wa[x], bk[hf][0], bk[hf][1]);
              mma_bf16_16816(acc(2 * hf + 1), wa[x], bk[hf][2], bk[hf][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (APART) S[4 * dp + i][c] += part[i][c];
      }
    }
#pragma unroll
    for (int nb = 0; nb < C / 8; ++nb)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = nb * 8 + 2 * tq + (i & 1), c = vcol + (i >> 1) * 8;
        if (t < cn && c < vdim) out[(row0 + t0 + t) * ((long long)H * vdim) + (long long)h * vdim + c] = APART ? o[nb][i] + (oh[nb][i] + ol[nb][i]) : o[nb][i];
      }
    __syncthreads();  // every warp is done with the tiles before the next block's are formed
  }
#pragma unroll
  for (int nb = 0; nb < DIM / 8; ++nb)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = nb * 8 + 2 * tq + (i & 1), c = vcol + (i >> 1) * 8;
      if (d < dim && c < vdim) stp[(long long)d * vdim + c] = S[nb][i];
    }
}

template <int DIM, int C, bool SILU, int CTAS>
int launch_blocks(const bf16* qkv, long long ld, float* state, const float* decay, float* out, const int* row0, const int* n, const int* ctx,
                  const int* slot, int entries, int H, int dim, int vdim, const PgLinearAttnOps& ops, cudaStream_t st) {
  const size_t smem = (size_t)(6 * C * (DIM + 8) + 3 * C * (C + 8) + (SILU ? 3 : 2) * C * 72) * sizeof(bf16) + (C + 1) * sizeof(float);
  auto kern = linear_attn_block_kernel<DIM, C, SILU, CTAS>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return PG_ERR_CUDA;
  pg::launch_spread(kern, dim3((vdim + 63) / 64, H, entries), 128, smem, st, qkv, ld, state, decay, out, row0, n, ctx, slot, H, dim, vdim, ops);
  pg_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}

}  // namespace

extern "C" int pg_linear_attn_blocks(const void* qkv, long long ld, float* state, const float* decay, float* out, const int* entry_row0,
                                     const int* entry_n, const int* entry_ctx, const int* entry_slot, int entries, int H, int dim, int vdim,
                                     const PgLinearAttnOps* options, void* stream) {
  if (entries <= 0 || entries > 65535 || H <= 0 || H > 65535 || options == nullptr) return PG_ERR_ARG;
  // 16-byte fetches of the rows, of the cosines and of the sines
  if (dim <= 0 || dim % 8 || dim > 128 || vdim <= 0 || vdim % 8 || ld % 8 || (reinterpret_cast<uintptr_t>(qkv) & 15)) return PG_ERR_ARG;
  if (!options->silu && options->rotate != nullptr && (2 * options->pairs < dim || options->pairs % 4 || (reinterpret_cast<uintptr_t>(options->rotate) & 15))) return PG_ERR_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // heads up to 64 wide with silu: three CTAs per SM (and a few spills) once there are more than two with tokens for each, else two (us, 2 / 3: 1536 CTAs 327 / 283, 384 of 300 tokens
  // 150 / 97, 288 84 / 102, 96 of 1500 tokens 279 / 310; without silu 1536 CTAs 187 / 202)
  const int portions = options->portions > 0 && options->portions < entries ? options->portions : entries;
  const bool many = (long long)((vdim + 63) / 64) * H * portions > 2LL * pg::num_sms();
#define PG_LB1(D, C, SILU, CTAS) \
  return launch_blocks<D, C, SILU, CTAS>(static_cast<const bf16*>(qkv), ld, state, decay, out, entry_row0, entry_n, entry_ctx, entry_slot, entries, H, dim, vdim, *options, st)
#define PG_LB(D, C, MANY)                            \
  do {                                               \
    if (options->silu && many) PG_LB1(D, C, true, MANY); \
    if (options->silu) PG_LB1(D, C, true, 2);        \
    PG_LB1(D, C, false, 2);                          \
  } while (0)
  if (dim <= 32) PG_LB(32, 32, 3);
  if (dim <= 64) PG_LB(64, 32, 3);
  if (dim <= 96) PG_LB(96, 32, 2);
  PG_LB(128, 32, 2);
#undef PG_LB1
#undef PG_LB
}
