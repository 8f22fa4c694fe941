// Steps (1) and (3) of the chunked recurrence of gated_recurrent.cu on the tensor cores, for a decay per channel, bfloat16 rows and no
// normaliser column: the 32-bit factors go in as three bfloat16 numbers each (split_mma.cuh), so nothing is lost against the FMA kernels.
// Included by gated_recurrent.cu, whose header has the formulas.
//
// (1): 22 us where the FMA kernel takes 53, (3): 58 us where it takes 117, for 2048 tokens and 16 heads of 128 x 128.  The heads' norm and gate in
// (3) are 4 and 15 us more (the gate's rows, four bytes a lane), which is what head_norm_gate takes for them and the rows' way there and back.
#pragma once
#include "split_mma.cuh"

// A chunk's log decays: thread (pair of channels, part of the tokens), in units of log 2.
template <int DP>
struct GmDecays {
  static constexpr int PAIRS = DP / 2, PARTS = 256 / PAIRS, TOK = GC / PARTS;
  float2 la[TOK];
  __device__ __forceinline__ void load(const float* __restrict__ log_decay, size_t t0, int n, int H, int h, int dim) {
    const int r = 2 * (threadIdx.x % PAIRS), i0 = threadIdx.x / PAIRS * TOK;
#pragma unroll
    for (int i = 0; i < TOK; ++i) {
      la[i] = make_float2(0.f, 0.f);
      if (r < dim && i0 + i < n) la[i] = __ldcg(reinterpret_cast<const float2*>(log_decay + ((t0 + i0 + i) * H + h) * dim + r));
    }
#pragma unroll
    for (int i = 0; i < TOK; ++i) la[i] = make_float2(la[i].x * GR_LOG2E, la[i].y * GR_LOG2E);
  }
  __device__ __forceinline__ float2 total() const {
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < TOK; ++i) s = make_float2(s.x + la[i].x, s.y + la[i].y);
    return s;
  }
};

// Values [GC][64 * TILES + 8] of bfloat16; rows from n on and columns from vdim on are zeros.
template <int COLS>
__device__ __forceinline__ void gm_load_values(bf16* dst, const bf16* __restrict__ v, size_t in_stride, int col0, int n, int vdim) {
#pragma unroll
  for (int idx = threadIdx.x; idx < GC * (COLS / 8); idx += 256) {
    const int i = idx / (COLS / 8), cc = idx % (COLS / 8) * 8;
    const bool here = i < n && col0 + cc < vdim;
    spl_cp16(dst + i * (COLS + 8) + cc, here ? v + i * in_stride + col0 + cc : v, here);
  }
}
// B fragments of 16 tokens and 16 columns; places 0 .. 3 of lane 4 g + t are tokens t, t + 4, t + 8, t + 12
template <int COLS>
__device__ __forceinline__ void gm_values_b(uint32_t (&b0)[2], uint32_t (&b1)[2], const bf16* v_s, int tok0, int col, int lane) {
  const int p = lane & 7, mat = lane >> 3;
  spl_ldmatrix_x4_trans(b0[0], b0[1], b1[0], b1[1], v_s + (tok0 + (p >> 1) + 4 * (p & 1) + 8 * (mat & 1)) * (COLS + 8) + col + 8 * (mat >> 1));
}

// (1): grid (S * H, chunks), 256 threads: a warp has 16 rows of the state; at DP = 64 two warps share the columns.
// The weighted keys lie in shared memory as [token][channel] in 32 bits and are split as they are read, once per row and column group.
// Bound: memory's round trips with two blocks an SM (a [dim, vdim] matrix a chunk leaves); the products are 6 us of it.
#define GM_COLS 128
template <int DP>
__global__ void __launch_bounds__(256, 2)
gated_mma_state_kernel(const bf16* __restrict__ k, const bf16* __restrict__ v, int in_stride, const float* __restrict__ log_decay,
                       const int* __restrict__ seq_start, float* __restrict__ scratch, float* __restrict__ chunk_decay, int max_chunks, int H,
                       int QH, int dim, int vdim) {
  using D = GmDecays<DP>;
  constexpr int LK = DP + 8;
  extern __shared__ __align__(16) float sm[];
  float* k_s = sm;                                        // [GC][LK]
  bf16* v_s = reinterpret_cast<bf16*>(k_s + GC * LK);     // [GC][GM_COLS + 8]
  __shared__ float2 tot[D::PARTS][D::PAIRS];
  pdl_trigger();
  pdl_wait();
  const int s = blockIdx.x / H, h = blockIdx.x % H, c = blockIdx.y, qh = h / (H / QH);
  const int t0 = __ldcg(seq_start + s) + c * GC;
  const int n = min(GC, __ldcg(seq_start + s + 1) - t0);
  if (n <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const bf16* vh = v + (size_t)t0 * in_stride + (size_t)h * vdim;
  gm_load_values<GM_COLS>(v_s, vh, in_stride, 0, n, vdim);
  spl_cp_commit();
  {
    const int pair = tid % D::PAIRS, part = tid / D::PAIRS, r = 2 * pair;
    uint32_t kv[D::TOK];
#pragma unroll
    for (int i = 0; i < D::TOK; ++i) {
      const int tok = part * D::TOK + i;
      kv[i] = 0u;
      if (r < dim && tok < n) kv[i] = __ldcg(reinterpret_cast<const uint32_t*>(k + (size_t)(t0 + tok) * in_stride + (size_t)qh * dim + r));
    }
    D d;
    d.load(log_decay, (size_t)t0, n, H, h, dim);
    tot[part][pair] = d.total();
    __syncthreads();
    float2 after = make_float2(0.f, 0.f);  // what the tokens after token i still take away
    for (int p = D::PARTS - 1; p > part; --p) after = make_float2(after.x + tot[p][pair].x, after.y + tot[p][pair].y);
#pragma unroll
    for (int i = D::TOK - 1; i >= 0; --i) {
      *reinterpret_cast<float2*>(k_s + (part * D::TOK + i) * LK + r) =
          make_float2(__uint_as_float(kv[i] << 16) * gr_exp2(after.x), __uint_as_float(kv[i] & 0xffff0000u) * gr_exp2(after.y));
      after = make_float2(after.x + d.la[i].x, after.y + d.la[i].y);
    }
    if (part == 0 && r < dim)
      *reinterpret_cast<float2*>(chunk_decay + ((size_t)blockIdx.x * max_chunks + c) * dim + r) = make_float2(gr_exp2(after.x), gr_exp2(after.y));
  }
  constexpr int ROW_WARPS = DP / 16, SHARE = GM_COLS * ROW_WARPS / 8;  // columns of a warp
  const int m0 = 16 * (warp % ROW_WARPS), n0 = warp / ROW_WARPS * SHARE;
  float* u = scratch + ((size_t)blockIdx.x * max_chunks + c) * dim * vdim;
  spl_cp_wait<0>();
  __syncthreads();
  SplA a[GC / 16];
#pragma unroll
  for (int kk = 0; kk < GC / 16; ++kk) {
    float lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float* at = k_s + (16 * kk + t + 4 * j) * LK + m0 + g;
      lo[j] = at[0];
      hi[j] = at[8];
    }
    spl_a(a[kk], lo, hi);
  }
#pragma unroll 1
  for (int nn = n0; nn < n0 + SHARE && nn < vdim; nn += 32) {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < GC / 16; ++kk) {
      uint32_t b[4][2];
      gm_values_b<GM_COLS>(b[0], b[1], v_s, 16 * kk, nn, lane);
      gm_values_b<GM_COLS>(b[2], b[3], v_s, 16 * kk, nn + 16, lane);
      spl_mma3_add<4>(acc, a[kk], b);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int col = nn + 8 * i + 2 * t;
      if (col < vdim) {
        if (m0 + g < dim) *reinterpret_cast<float2*>(u + (size_t)(m0 + g) * vdim + col) = make_float2(acc[i][0], acc[i][1]);
        if (m0 + g + 8 < dim) *reinterpret_cast<float2*>(u + (size_t)(m0 + g + 8) * vdim + col) = make_float2(acc[i][2], acc[i][3]);
      }
    }
  }
}

// Eight products' sums over the warp, one to four lanes each: lane 4 j + x ends with the sum of s[j].
__device__ __forceinline__ float gm_sum8(float (&s)[8], int lane) {
#pragma unroll
  for (int o = 4; o >= 1; o >>= 1) {  // half of what is left goes to the lane 4 o away, whose other half comes here
    const bool upper = lane & (4 * o);
#pragma unroll
    for (int e = 0; e < o; ++e) {
      const float give = upper ? s[e] : s[e + o], keep = upper ? s[e + o] : s[e];
      s[e] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * o);
    }
  }
  s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
  s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
  return s[0];
}

// (3): grid (S * H, chunks), 256 threads, two blocks an SM.
// Scores.  With A_i the running sum of the log decays, a pair i > j of different eights of tokens factors at a border b between them,
// exp(A_i - A_j) = exp(A_i - A_b) exp(A_b - A_j), both exponents <= 0 whatever the decays are: b = 31 for the lower left quarter of the
// chunk (four warps), 15 and 47 for those of its halves (two warps), 7, 23, 39 and 55 for those of their halves (two warps, two of them to
// an instruction).  So each warp makes the fragments of its products from the rows and the sums as it loads them, 12 instructions of
// m16n8k16 for 16 channels.  Pairs within eight tokens take an exponential per channel: a warp per eight, a lane four channels.
// Outputs.  (scores) x (values, bfloat16: three products) and (queries times exp(A_i)) x (state: six); a warp has all 64 tokens and 16
// columns, so that the state, split as it is read, is split once.  Scores and queries are kept as their three parts and come by ldmatrix;
// the queries' parts take the place of the sums and the scores, the state's halves (eight columns of every warp) that of q and k.
// With a norm the heads' norm and gate are applied before the result leaves (the sums of squares meet in shared memory): a pass over
// 32-bit rows less than head_norm_gate behind it, with the same bits.
// Bound: of a block's 42000 cycles (two share the SM, in step) the loads take 7000, the scores 15000 (exponentials and splits: issue slots)
// and the outputs 16000, which is what the tensor cores' legacy instruction takes there (4320 a block, 3072 of them the queries against the
// state).  With operands split by every warp that reads them, from 32-bit tiles of 64 columns, it was 65 us instead of 58.
template <int DP>
struct GmOut {
  static constexpr int LQ = DP + 16, LA = DP + 4, LP = DP + 8, LS = 68, LV = 128 + 8;
  static constexpr int X = GC * LQ * 4 > DP * LS * 4 ? GC * LQ * 4 : DP * LS * 4;
  static constexpr int SUMS = GC * LA * 4, MIDDLE = SUMS + 3 * SPL_TRI_BYTES > 3 * GC * LP * 2 ? SUMS + 3 * SPL_TRI_BYTES : 3 * GC * LP * 2;
  static constexpr int BYTES = X + MIDDLE + GC * LV * 2;
};
__device__ __forceinline__ void gm_four(float (&f)[4], const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
  f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
}
// v *= exp2(plus - minus), four channels
__device__ __forceinline__ void gm_decay4(float (&v)[4], const float* plus, const float* minus) {
  const float4 p = *reinterpret_cast<const float4*>(plus), m = *reinterpret_cast<const float4*>(minus);
  v[0] *= gr_exp2(p.x - m.x);
  v[1] *= gr_exp2(p.y - m.y);
  v[2] *= gr_exp2(p.z - m.z);
  v[3] *= gr_exp2(p.w - m.w);
}
template <int DP>
__global__ void __launch_bounds__(256, 2)
gated_mma_out_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v, int in_stride,
                     const float* __restrict__ log_decay, float q_scale, const int* __restrict__ seq_start, const float* __restrict__ scratch,
                     int max_chunks, void* __restrict__ out, int out_stride, int H, int QH, int dim, int vdim, SplNorm norm) {
  using D = GmDecays<DP>;
  using L = GmOut<DP>;
  constexpr int LQ = L::LQ, LA = L::LA, LP = L::LP, LS = L::LS, LV = L::LV;
  extern __shared__ __align__(16) unsigned char gm_smem[];
  bf16* q_s = reinterpret_cast<bf16*>(gm_smem);                    // [GC][LQ]
  bf16* k_s = q_s + GC * LQ;                                       // [GC][LQ]
  float* s_s = reinterpret_cast<float*>(gm_smem);                  // [DP][LS], later
  float* a_s = reinterpret_cast<float*>(gm_smem + L::X);           // [GC][LA]: the sums A_i
  unsigned char* p_s = gm_smem + L::X + L::SUMS;                   // [3][10 tiles]: the scores' parts
  bf16* qp_s = reinterpret_cast<bf16*>(gm_smem + L::X);            // [3][GC][LP]: the decayed queries' parts, later
  bf16* v_s = reinterpret_cast<bf16*>(gm_smem + L::X + L::MIDDLE); // [GC][LV]
  __shared__ __align__(16) float2 tot[D::PARTS][D::PAIRS];
  pdl_trigger();
  pdl_wait();
  const int s = blockIdx.x / H, h = blockIdx.x % H, c = blockIdx.y, qh = h / (H / QH);
  const int t0 = __ldcg(seq_start + s) + c * GC;
  const int n = min(GC, __ldcg(seq_start + s + 1) - t0);
  if (n <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  for (int idx = tid; idx < GC * (DP / 8); idx += 256) {
    const int i = idx / (DP / 8), r = idx % (DP / 8) * 8;
    const bool here = i < n && r < dim;
    const size_t at = (size_t)(t0 + i) * in_stride + (size_t)qh * dim + r;
    spl_cp16(q_s + i * LQ + r, here ? q + at : q, here);
    spl_cp16(k_s + i * LQ + r, here ? k + at : k, here);
  }
  gm_load_values<128>(v_s, v + (size_t)t0 * in_stride + (size_t)h * vdim, in_stride, 0, n, vdim);
  spl_cp_commit();
  {
    const int pair = tid % D::PAIRS, part = tid / D::PAIRS;
    D d;
    d.load(log_decay, (size_t)t0, n, H, h, dim);
    tot[part][pair] = d.total();
    __syncthreads();
    float2 run = make_float2(0.f, 0.f);
    for (int p = 0; p < part; ++p) run = make_float2(run.x + tot[p][pair].x, run.y + tot[p][pair].y);
#pragma unroll
    for (int i = 0; i < D::TOK; ++i) {
      run = make_float2(run.x + d.la[i].x, run.y + d.la[i].y);
      *reinterpret_cast<float2*>(a_s + (part * D::TOK + i) * LA + 2 * pair) = run;
    }
  }
  spl_cp_wait<0>();
  __syncthreads();
  auto put_scores = [&](int i, int j, float x, float y) { spl_tri_put(p_s, i, j, x, y); };
  // ---- scores between eights
  {
    // rows g and g + 8 of the instruction's A and its two groups of eight keys: first token, and the border they meet at
    int row_lo, row_hi, border_lo, border_hi, key0, key1;
    if (warp < 4) {
      row_lo = 32 + 16 * (warp & 1), row_hi = row_lo + 8, border_lo = border_hi = 31, key0 = 16 * (warp >> 1), key1 = key0 + 8;
    } else if (warp < 6) {
      const int b = 32 * (warp - 4);
      row_lo = b + 16, row_hi = b + 24, border_lo = border_hi = b + 15, key0 = b, key1 = b + 8;
    } else {
      const int b = 32 * (warp - 6);
      row_lo = b + 8, row_hi = b + 24, border_lo = b + 7, border_hi = b + 23, key0 = b, key1 = b + 16;
    }
    float acc[1][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) acc[0][i][0] = acc[0][i][1] = acc[0][i][2] = acc[0][i][3] = 0.f;
#pragma unroll 1
    for (int kk = 0; kk < DP / 16; ++kk) {
      const int r = 16 * kk + 4 * t;
      float lo[4], hi[4], y0[4], y1[4];
      gm_four(lo, q_s + (row_lo + g) * LQ + r);
      gm_four(hi, q_s + (row_hi + g) * LQ + r);
      gm_four(y0, k_s + (key0 + g) * LQ + r);
      gm_four(y1, k_s + (key1 + g) * LQ + r);
      gm_decay4(lo, a_s + (row_lo + g) * LA + r, a_s + border_lo * LA + r);
      gm_decay4(hi, a_s + (row_hi + g) * LA + r, a_s + border_hi * LA + r);
      gm_decay4(y0, a_s + border_lo * LA + r, a_s + (key0 + g) * LA + r);
      gm_decay4(y1, a_s + border_hi * LA + r, a_s + (key1 + g) * LA + r);
      SplA a[1];
      SplB b[2];
      spl_a(a[0], lo, hi);
      spl_b(b[0], y0);
      spl_b(b[1], y1);
      spl_mma6_add<1, 2>(acc, a, b);
    }
    put_scores(row_lo + g, key0 + 2 * t, acc[0][0][0] * q_scale, acc[0][0][1] * q_scale);
    put_scores(row_hi + g, key1 + 2 * t, acc[0][1][2] * q_scale, acc[0][1][3] * q_scale);
    if (warp < 6) {  // (else rows g belong to the first keys only, rows g + 8 to the second)
      put_scores(row_lo + g, key1 + 2 * t, acc[0][1][0] * q_scale, acc[0][1][1] * q_scale);
      put_scores(row_hi + g, key0 + 2 * t, acc[0][0][2] * q_scale, acc[0][0][3] * q_scale);
    }
  }
  // ---- scores within eight tokens: a decay per channel; a token with itself has none
  {
    const int i0 = 8 * warp, r = 4 * lane;
    float ka[8][4], kk[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (r < DP) {
        gm_four(kk[i], k_s + (i0 + i) * LQ + r);
        const float4 a = *reinterpret_cast<const float4*>(a_s + (i0 + i) * LA + r);
        ka[i][0] = a.x, ka[i][1] = a.y, ka[i][2] = a.z, ka[i][3] = a.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) kk[i][e] = ka[i][e] = 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float x[4] = {0.f, 0.f, 0.f, 0.f}, sum[8];
      if (r < DP) gm_four(x, q_s + (i0 + i) * LQ + r);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        sum[j] = 0.f;
        if (j < i) {
#pragma unroll
          for (int e = 0; e < 4; ++e) sum[j] = fmaf(x[e] * kk[j][e], gr_exp2(ka[i][e] - ka[j][e]), sum[j]);
        } else if (j == i) {
#pragma unroll
          for (int e = 0; e < 4; ++e) sum[j] = fmaf(x[e], kk[j][e], sum[j]);
        }
      }
      const float mine = gm_sum8(sum, lane) * q_scale, next = __shfl_down_sync(0xffffffffu, mine, 4);
      const int j = lane >> 2;  // (later tokens' sums are zeros)
      if ((lane & 7) == 0) put_scores(i0 + i, i0 + j, mine, next);
      if ((warp & 1) == 0 && (lane & 7) == 1) put_scores(i0 + i, i0 + 8 + j, 0.f, 0.f);  // the later half of the tile of 16
    }
  }
  // ---- the queries against the state before the chunk take the whole decay since the chunk's start
  constexpr int PER = GC * DP / 4 / 256;
  float x[PER][4];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int idx = tid + 256 * p, i = idx / (DP / 4), r = idx % (DP / 4) * 4;
    gm_four(x[p], q_s + i * LQ + r);
    const float4 a = *reinterpret_cast<const float4*>(a_s + i * LA + r);
    x[p][0] *= q_scale * gr_exp2(a.x);
    x[p][1] *= q_scale * gr_exp2(a.y);
    x[p][2] *= q_scale * gr_exp2(a.z);
    x[p][3] *= q_scale * gr_exp2(a.w);
  }
  __syncthreads();  // the scores are there; q, k and the sums are used up
  const float* sp = scratch + ((size_t)blockIdx.x * max_chunks + c) * dim * vdim;
  auto load_state = [&](int half) {  // columns 16 w + 8 half .. of every warp w
#pragma unroll 4
    for (int idx = tid; idx < DP * 16; idx += 256) {
      const int r = idx >> 4, e = idx & 15, col = 16 * (e >> 1) + 8 * half + 4 * (e & 1);
      const bool here = r < dim && col < vdim;
      spl_cp16(s_s + r * LS + 4 * e, here ? sp + (size_t)r * vdim + col : sp, here);
    }
    spl_cp_commit();
  };
  load_state(0);
  float acc[2][2][2][1][4] = {};  // [half][32 tokens][16 of them]
#pragma unroll
  for (int kt = 0; kt < GC / 16; ++kt) {
    uint32_t b[2][2];
    spl_ldmatrix_x4_trans(b[0][0], b[0][1], b[1][0], b[1][1], v_s + (16 * kt + (lane & 15)) * LV + 16 * warp + 8 * (lane >> 4));
#pragma unroll
    for (int m = kt; m < 4; ++m) {
      SplA a;
      spl_tri_a(a, p_s, m, kt, lane);
      float d[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) spl_mma_zero(d[i], a.p[2], b[i]);
#pragma unroll
      for (int i = 0; i < 2; ++i) spl_mma(d[i], a.p[1], b[i]);
#pragma unroll
      for (int i = 0; i < 2; ++i) spl_mma(d[i], a.p[0], b[i]);
#pragma unroll
      for (int i = 0; i < 2; ++i) spl_add(acc[i][m >> 1][m & 1][0], d[i]);
    }
  }
  __syncthreads();  // the scores are used up
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int idx = tid + 256 * p, i = idx / (DP / 4), r = idx % (DP / 4) * 4;
    uint2 w[3];
    spl_pair(x[p][0], x[p][1], w[0].x, w[1].x, w[2].x);
    spl_pair(x[p][2], x[p][3], w[0].y, w[1].y, w[2].y);
#pragma unroll
    for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(qp_s + (e * GC + i) * LP + r) = w[e];
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    if (half) {
      __syncthreads();  // the first half is used up
      load_state(1);
    }
    spl_cp_wait<0>();
    __syncthreads();
    if (16 * warp + 8 * half < vdim) {
#pragma unroll 1
      for (int kk = 0; kk < DP / 16; ++kk) {
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = s_s[(16 * kk + 2 * t + (e & 1) + 8 * (e >> 1)) * LS + 8 * warp + g];
        SplB b[1];
        spl_b(b[0], y);
#pragma unroll
        for (int mm = 0; mm < 4; mm += 2) {
          SplA a[2];
#pragma unroll
          for (int m = 0; m < 2; ++m) spl_rows_a(a[m], qp_s + 16 * (mm + m) * LP + 16 * kk, GC * LP, LP, lane);
          spl_mma6_add<2, 1>(acc[half][mm / 2], a, b);
        }
      }
    }
  }
  spl_finish(acc, reinterpret_cast<float*>(gm_smem), n, t0, h, vdim, 0, out, out_stride, norm);
}

// Sizes and addresses that these kernels take: rows in whole 16-byte pieces, keys and values up to 128.  (That the state's, the scratch's and the
// output's rows are whole 16-byte pieces is GC_WIDE_STATE's to say.)
static inline bool gated_mma_takes(const void* q, const void* k, const void* v, int in_stride, const float* log_decay, int dim, int vdim) {
  return dim <= 128 && vdim <= 128 && dim % 8 == 0 && vdim % 8 == 0 && in_stride % 8 == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)log_decay) & 15) == 0;
}
