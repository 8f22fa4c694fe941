// The gated delta rule for prompts of a bfloat16 run, chunk by chunk instead of token by token (delta_rule.cu has the rule and the
// token-by-token kernel, which takes single tokens, short portions and 32-bit runs).
//
// Inside a chunk of 64 tokens, with L_i the sum of the log decays up to token i and S_0 the state before the chunk,
//
//     S_i = e^(L_i) S_0 + sum_(j <= i) e^(L_i - L_j) k_j u_j^T,      u_i = beta_i (v_i - e^(L_i) S_0^T k_i - sum_(j < i) e^(L_i - L_j) (k_i . k_j) u_j)
//
// so the u of a chunk solve a unit triangular system (I + A) U = diag(beta) (V - diag(e^L) K S_0), A_ij = beta_i e^(L_i - L_j) (k_i . k_j)
// for j < i, and with  T = (I + A)^-1 diag(beta),  X = T V  and  W = T diag(e^L) K  they are U = X - W S_0.  (T's entries stay small: it is
// made of products of contractions, I - beta k k^T of a unit vector k.)  Decays only enter as e to the difference of two sums where the
// difference is not positive: nothing overflows, what underflows is zero.
//
//   (1) delta_chunk_solve   per (chunk, head): A, T by blocks, X and W; leaves W and the keys split into three bfloat16 parts
//   (2) delta_chunk_walk    per (32 or 16 columns of the state, head, sequence), chunk after chunk: U = X - W S, S <- e^(L_63) S + K^T (e^(L_63 - L) U);
//                           leaves U in X's place and the state before every chunk
//   (3) delta_chunk_out     per (chunk, head): O = diag(e^L) Q S_0 + (Q K^T * e^(L_i - L_j), j <= i) U, and the head's norm where it is asked for
//
// All operands are 32-bit (but for the values) and go to the tensor cores as three bfloat16 numbers each, which loses no digits against
// FMAs (split_mma.cuh).  Token by token every token is one chain of dependent steps per column; here only (2) is serial, with 64 tokens a
// step.  Sequences of 1029, 700 and 319 tokens, 16 heads of 128 x 128: 53, 80 and 58 us (78 with the heads' norm and gate); by FMAs fed from shared
// memory 62, 106 and 72 (and 17 for norm and gate), token by token 444.
#include "split_mma.cuh"

RL_DEFINE_ERROR_TEXT()

#define DC 64  // tokens per chunk

// The chunks that one go of the three steps works on, and their places in the scratch.  All of them at once (count 0): those of sequence s
// start at seq_start[s] / 64 + s (room for every sequence's last, partly filled one).  Where the scratch is smaller, `count` of every sequence at
// a time, from its chunk `first` on: the state goes from one go to the next in the sequences' records, the same 32 bits as in registers.
struct DcWindow {
  int first, count;
};
__device__ __forceinline__ int dc_chunk(const DcWindow& w, int start, int s, int c) { return w.count ? s * w.count + c - w.first : start / DC + s + c; }

// Running sums of 64 log decays (zero past the chunk's last token) by one warp, two to a lane.  In 64 bits: what is used of them are
// differences, and those of fast decays are small beside the sums.  A log decay may be minus infinity, whose differences are no numbers:
// from DC_LOG_LEAST down, where the exponential has long been zero, all are the same.
#define DC_LOG_LEAST (-16384.f)
__device__ __forceinline__ double dc_log(const float* __restrict__ log_decay) {
  const float l = __ldcg(log_decay);
  return (double)(l < DC_LOG_LEAST ? DC_LOG_LEAST : l);  // (what is no number stays so)
}
__device__ __forceinline__ void dc_log_sums(const float* __restrict__ log_decay, int t0, int n, int H, int h, double* L, int lane) {
  const double a = 2 * lane < n ? dc_log(log_decay + (size_t)(t0 + 2 * lane) * H + h) : 0.0;
  const double b = 2 * lane + 1 < n ? dc_log(log_decay + (size_t)(t0 + 2 * lane + 1) * H + h) : 0.0;
  double run = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += v;
  }
  const double before = __shfl_up_sync(0xffffffffu, run, 1);
  const double base = lane ? before : 0.0;
  L[2 * lane] = base + a;
  L[2 * lane + 1] = base + (a + b);
}
__device__ __forceinline__ float dc_decay(double later, double earlier) { return expf((float)(later - earlier)); }

// The parts of 64 rows of up to DP numbers, [3][64][DP]: pieces of eight numbers stand where their number in the row, turned by the row's,
// says, so that the same piece of eight rows lies in different banks.  In scratch as in shared memory: a tile moves as it is.
template <int DP>
__device__ __forceinline__ int dc_at(int row, int piece) { return row * DP + ((piece ^ (row & 7)) << 3); }
// A row's eight numbers from 32 bits into their three parts
template <int DP>
__device__ __forceinline__ void dc_put8(bf16* parts, int row, int piece, const float4& x, const float4& y) {
  uint4 p[3];
  spl_pair(x.x, x.y, p[0].x, p[1].x, p[2].x);
  spl_pair(x.z, x.w, p[0].y, p[1].y, p[2].y);
  spl_pair(y.x, y.y, p[0].z, p[1].z, p[2].z);
  spl_pair(y.z, y.w, p[0].w, p[1].w, p[2].w);
#pragma unroll
  for (int e = 0; e < 3; ++e) *reinterpret_cast<uint4*>(parts + e * DC * DP + dc_at<DP>(row, piece)) = p[e];
}
// 64 rows of dim numbers in 32 bits, `ld` apart (rows from n on and columns from dim on are zeros): a thread's share, all of it asked for at once
template <int DP>
struct DcRows {
  static constexpr int PER = DC * DP / 8 / 256;
  float4 x[PER], y[PER];
  __device__ __forceinline__ static int row(int p) { return (threadIdx.x + 256 * p) / (DP / 8); }
  __device__ __forceinline__ static int piece(int p) { return (threadIdx.x + 256 * p) % (DP / 8); }
  __device__ __forceinline__ void load(const float* __restrict__ src, size_t ld, int n, int dim) {
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int r = row(p), k = 8 * piece(p);
      const float* at = src + r * ld + k;
      x[p] = r < n && k < dim ? __ldcg(reinterpret_cast<const float4*>(at)) : make_float4(0.f, 0.f, 0.f, 0.f);
      y[p] = r < n && k + 4 < dim ? __ldcg(reinterpret_cast<const float4*>(at + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
};
// A tile of parts from scratch into shared memory
template <int DP>
__device__ __forceinline__ void dc_load_parts(bf16* dst, const bf16* __restrict__ src) {
#pragma unroll
  for (int i = 0; i < 3 * DC * DP / 8 / 256; ++i) spl_cp16(dst + 8 * (threadIdx.x + 256 * i), src + 8 * (threadIdx.x + 256 * i), true);
}
// 16 rows from m0 and 16 of k from 16 kk on as an A operand
template <int DP>
__device__ __forceinline__ void dc_a(SplA& a, const bf16* parts, int m0, int kk, int lane) {
  const bf16* at = parts + dc_at<DP>(m0 + (lane & 15), 2 * kk + (lane >> 4));
#pragma unroll
  for (int e = 0; e < 3; ++e) spl_ldmatrix_x4(a.p[e][0], a.p[e][1], a.p[e][2], a.p[e][3], at + e * DC * DP);
}

// The lower triangle of x y^T, 64 rows of DP numbers each, in pieces of 16 rows and 8 columns: warp w < 4 has the first half of row piece w,
// warp 4 + w the second half of row piece 3 - w, so that every quarter of the SM has five of them.
template <int DP, int NT>
__device__ __forceinline__ void dc_inner_row(float (&sum)[4][4], const bf16* x, const bf16* y, int m, int first, int lane) {
  constexpr int PAIRS = (NT + 1) / 2;
  float acc[1][NT][4] = {};
#pragma unroll 2
  for (int kk = 0; kk < DP / 16; ++kk) {
    SplA a[1];
    SplB b[2 * PAIRS];
    dc_a<DP>(a[0], x, 16 * m, kk, lane);
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
      const bf16* at = y + dc_at<DP>(8 * (first + 2 * i) + 8 * (lane >> 4) + (lane & 7), 2 * kk + ((lane >> 3) & 1));
#pragma unroll
      for (int e = 0; e < 3; ++e)
        spl_ldmatrix_x4(b[2 * i].p[e][0], b[2 * i].p[e][1], b[2 * i + 1].p[e][0], b[2 * i + 1].p[e][1], at + e * DC * DP);
    }
    spl_mma6_add<1, NT>(acc, a, reinterpret_cast<const SplB(&)[NT]>(b));
  }
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[i][e] = acc[0][i][e];
}
template <int DP>
__device__ __forceinline__ void dc_inner_lower(float (&sum)[4][4], const bf16* x, const bf16* y, int warp, int lane) {
  const int m = warp < 4 ? warp : 7 - warp, first = warp < 4 ? 0 : m + 1;
  if (m == 0) dc_inner_row<DP, 1>(sum, x, y, 0, first, lane);
  else if (m == 1) dc_inner_row<DP, 2>(sum, x, y, 1, first, lane);
  else if (m == 2) dc_inner_row<DP, 3>(sum, x, y, 2, first, lane);
  else dc_inner_row<DP, 4>(sum, x, y, 3, first, lane);
}
// every pair of neighbouring numbers of it
template <typename F>
__device__ __forceinline__ void dc_inner_each(const float (&sum)[4][4], int warp, int lane, F&& use) {
  const int m = warp < 4 ? warp : 7 - warp, first = warp < 4 ? 0 : m + 1, row = 16 * m + (lane >> 2);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (i <= m) {
      const int col = 8 * (first + i) + 2 * (lane & 3);
      use(row, col, sum[i][0], sum[i][1]);
      use(row + 8, col, sum[i][2], sum[i][3]);
    }
}

// What a row does not see must not reach it: in a tile on the diagonal a zero stands before later tokens' numbers, and zero times what is no
// number is none.  So there such numbers are taken out of the product (`parts` registers hold two each of this lane's column, the first of
// which shows what they are), and `first` becomes their first row in that column (16: there is none).
__device__ __forceinline__ bool dc_no_number(uint32_t half) { return (half & 0x7f80u) == 0x7f80u; }
template <int PARTS>
__device__ __forceinline__ bool dc_take_out(uint32_t (*b)[2], int& first, int t) {
  first = 16;
  bool any = false;
#pragma unroll
  for (int r = 0; r < 2; ++r) any |= dc_no_number(b[0][r]) || dc_no_number(b[0][r] >> 16);
  if (!__any_sync(0xffffffffu, any)) return false;
#pragma unroll
  for (int r = 1; r >= 0; --r) {
    const bool low = dc_no_number(b[0][r]), high = dc_no_number(b[0][r] >> 16);
    if (high) first = 8 * r + 2 * t + 1;
    if (low) first = 8 * r + 2 * t;
#pragma unroll
    for (int e = 0; e < PARTS; ++e) b[e][r] &= (low ? 0xffff0000u : 0xffffffffu) & (high ? 0xffffu : 0xffffffffu);
  }
  first = min(first, __shfl_xor_sync(0xffffffffu, first, 1));
  first = min(first, __shfl_xor_sync(0xffffffffu, first, 2));
  return true;
}
__device__ __forceinline__ void dc_put_back(float (&acc)[4], int first, int g, int t) {
  const float none = __int_as_float(0x7fffffff);
  const int f0 = __shfl_sync(0xffffffffu, first, 8 * t), f1 = __shfl_sync(0xffffffffu, first, 8 * t + 4);
  if (g >= f0) acc[0] = none;
  if (g >= f1) acc[1] = none;
  if (g + 8 >= f0) acc[2] = none;
  if (g + 8 >= f1) acc[3] = none;
}

// ---------------------------------------------------------------- (1)
// T by halves: the inverses of eight diagonal blocks of 8 x 8 by substitution (a thread a column), then twice, four and eight times that size
// by  [T1 0; -T2 A21 T1  T2].  Then a warp has 16 columns of X, and after that of W.
// A token whose key, strength or decay is no number: the tokens before it are as if there were nothing after, it and all later ones have no
// number (their u, and with them the state, could have none).
// Operands are split once, where they are loaded or made, and come to the tensor cores by ldmatrix: with every warp splitting what it read,
// and W's parts leaving four bytes at a time from the sums' lanes, the kernel took as long as the FMAs'.
template <int DP>
struct DcSolve {
  static constexpr int LA = 72, LV = 136;
  static constexpr int PARTS = 3 * DC * DP * 2;
  static constexpr int BYTES = PARTS + 2 * DC * LA * 4 + DC * LV * 2;
};
template <int N>
struct DcFloats;
template <>
struct DcFloats<1> { typedef float type; };
template <>
struct DcFloats<2> { typedef float2 type; };
template <>
struct DcFloats<4> { typedef float4 type; };
// acc[e] += f * at[e] for N neighbouring floats of shared memory
template <int N>
__device__ __forceinline__ void dc_axpy(float (&acc)[N], float f, const float* at) {
  float v[N];
  *reinterpret_cast<typename DcFloats<N>::type*>(v) = *reinterpret_cast<const typename DcFloats<N>::type*>(at);
#pragma unroll
  for (int e = 0; e < N; ++e) acc[e] = fmaf(f, v[e], acc[e]);
}
template <int N>
__device__ __forceinline__ void dc_widen(const float* a_s, float* t_s) {  // thread: a row of the 32 that have a block to their left, and N of its columns
  constexpr int B = 8 * N, LA = 72;
  const int row = threadIdx.x >> 3, r = row % B, base = row / B * 2 * B, col = (threadIdx.x & 7) * N;
  float* to = t_s + (base + B + r) * LA + base + col;
  float x[N];
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {  // A21 T1, then -T2 of it
    const float* left = pass ? t_s + (base + B + r) * LA + base + B : a_s + (base + B + r) * LA + base;
    const float* right = t_s + (pass ? base + B : base) * LA + base + col;
#pragma unroll
    for (int e = 0; e < N; ++e) x[e] = 0.f;
#pragma unroll
    for (int k = 0; k < B; k += 4) {
      const float4 f = *reinterpret_cast<const float4*>(left + k);
      dc_axpy<N>(x, f.x, right + k * LA);
      dc_axpy<N>(x, f.y, right + (k + 1) * LA);
      dc_axpy<N>(x, f.z, right + (k + 2) * LA);
      dc_axpy<N>(x, f.w, right + (k + 3) * LA);
    }
    if (pass) __syncthreads();
#pragma unroll
    for (int e = 0; e < N; ++e) to[e] = pass ? -x[e] : x[e];
    __syncthreads();
  }
}

template <int DP>
__global__ void __launch_bounds__(256, 2)
delta_chunk_solve_kernel(const float* __restrict__ kn, const bf16* __restrict__ v, int v_stride, int v_wide, const float* __restrict__ beta,
                         const float* __restrict__ log_decay, const int* __restrict__ seq_start, bf16* __restrict__ W, bf16* __restrict__ K,
                         float* __restrict__ U, float* __restrict__ tails, int H, int G, int dim, int vdim, int min_len, DcWindow win) {
  extern __shared__ __align__(16) unsigned char dc_smem[];
  constexpr int LA = DcSolve<DP>::LA, LV = DcSolve<DP>::LV;
  bf16* k_s = reinterpret_cast<bf16*>(dc_smem);                             // the keys' parts, then W's
  float* a_s = reinterpret_cast<float*>(dc_smem + DcSolve<DP>::PARTS);      // [64][LA]: A
  unsigned char* tri = reinterpret_cast<unsigned char*>(a_s);               // then T's parts
  float* t_s = a_s + DC * LA;                                               // [64][LA]: (I + A)^-1
  bf16* v_s = reinterpret_cast<bf16*>(t_s + DC * LA);                       // [64][LV]
  __shared__ double L[DC];
  __shared__ __align__(8) float be[DC], from_start[DC];
  __shared__ int good;  // tokens before the first whose numbers are none
  pdl_trigger();
  pdl_wait();
  const int c = win.first + blockIdx.x, h = blockIdx.y, s = blockIdx.z, kh = h / (H / G), tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int start = __ldcg(seq_start + s), end = __ldcg(seq_start + s + 1), t0 = start + c * DC;
  const int n = min(DC, end - t0);
  if (n <= 0 || end - start < min_len) return;
  const bf16* vh = v + (size_t)t0 * v_stride + (size_t)h * vdim;
  auto load_values = [&](int col0) {
    if (v_wide) {
      for (int idx = tid; idx < DC * 16; idx += 256) {
        const int i = idx >> 4, cc = (idx & 15) * 8;
        const bool here = i < n && col0 + cc < vdim;
        spl_cp16(v_s + i * LV + cc, here ? vh + (size_t)i * v_stride + col0 + cc : v, here);
      }
    } else {
      for (int idx = tid; idx < DC * 128; idx += 256) {
        const int i = idx >> 7, cc = idx & 127;
        v_s[i * LV + cc] = i < n && col0 + cc < vdim ? __ldcg(vh + (size_t)i * v_stride + col0 + cc) : __float2bfloat16_rn(0.f);
      }
    }
    spl_cp_commit();
  };
  DcRows<DP> rows;
  rows.load(kn + ((size_t)t0 * G + kh) * dim, (size_t)G * dim, n, dim);
  load_values(0);
  if (tid < 32) dc_log_sums(log_decay, t0, n, H, h, L, tid);
  if (tid >= 64 && tid < 64 + DC) be[tid - 64] = tid - 64 < n ? __ldcg(beta + (size_t)(t0 + tid - 64) * H + h) : 0.f;
  if (tid == 255) good = DC;
  for (int i = tid; i < DC * LA / 4; i += 256) reinterpret_cast<float4*>(t_s)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  {
    int bad = DC;
#pragma unroll
    for (int p = 0; p < DcRows<DP>::PER; ++p) {
      const float4 x = rows.x[p], y = rows.y[p];
      if (((x.x * 0.f + x.y * 0.f) + (x.z * 0.f + x.w * 0.f)) + ((y.x * 0.f + y.y * 0.f) + (y.z * 0.f + y.w * 0.f)) != 0.f) bad = min(bad, rows.row(p));
      dc_put8<DP>(k_s, rows.row(p), rows.piece(p), x, y);
    }
    if (tid < DC && (be[tid] * 0.f != 0.f || L[tid] * 0.0 != 0.0)) bad = min(bad, tid);
    if (bad < DC) atomicMin(&good, bad);
  }
  __syncthreads();
  const int ok = good;
  const size_t chunk = dc_chunk(win, start, s, c), slot = chunk * H + h;
  if (h % (H / G) == 0) {  // the keys' parts, once for the heads that share them
    uint4* to = reinterpret_cast<uint4*>(K + (chunk * G + kh) * 3 * DC * DP);
#pragma unroll 4
    for (int i = tid; i < 3 * DC * DP / 8; i += 256) to[i] = reinterpret_cast<const uint4*>(k_s)[i];
  }
  if (ok < DC) {
    __syncthreads();
    for (int i = tid; i < 3 * DC * DP / 8; i += 256)
      if (i / (DP / 8) % DC >= ok) reinterpret_cast<uint4*>(k_s)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid >= ok && tid < DC) be[tid] = 0.f;
    __syncthreads();
  }
  if (tid < DC) {
    from_start[tid] = tid < ok ? dc_decay(L[tid], 0.0) : 0.f;
    // what is left of a token's write, and of the state before the chunk, at the chunk's end
    tails[slot * (DC + 4) + tid] = dc_decay(L[DC - 1], L[tid]);
    if (tid == 0) tails[slot * (DC + 4) + DC] = dc_decay(L[DC - 1], 0.0);
  }
  float inner[4][4];
  dc_inner_lower<DP>(inner, k_s, k_s, warp, lane);
  dc_inner_each(inner, warp, lane, [&](int i, int j, float x, float y) {
    const bool seen = i < ok;
    *reinterpret_cast<float2*>(a_s + i * LA + j) =
        make_float2(seen && j < i ? be[i] * dc_decay(L[i], L[j]) * x : 0.f, seen && j + 1 < i ? be[i] * dc_decay(L[i], L[j + 1]) * y : 0.f);
  });
  __syncthreads();
  // ---- the inverse
  if (tid < DC) {
    const int b = tid & ~7, col = tid & 7;
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[i] = i == col ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) x[i] = fmaf(-a_s[(b + i) * LA + b + j], x[j], x[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) t_s[(b + i) * LA + b + col] = x[i];
  }
  __syncthreads();
  dc_widen<1>(a_s, t_s);
  dc_widen<2>(a_s, t_s);
  dc_widen<4>(a_s, t_s);
  // ---- X, then W: T's parts with the factors of its columns, tile by tile times 16 columns of a warp
  auto put_t = [&](bool of_w) {
#pragma unroll
    for (int p = 0; p < 5; ++p) {
      const int idx = tid + 256 * p, tile = idx >> 7, m = tile < 1 ? 0 : tile < 3 ? 1 : tile < 6 ? 2 : 3, kt = tile - m * (m + 1) / 2;
      const int i = 16 * m + ((idx >> 3) & 15), j = 16 * kt + 2 * (idx & 7);
      const float2 x = *reinterpret_cast<const float2*>(t_s + i * LA + j);
      float2 f = *reinterpret_cast<const float2*>(be + j);
      if (of_w) f = make_float2(f.x * from_start[j], f.y * from_start[j + 1]);
      spl_tri_put(tri, i, j, x.x * f.x, x.y * f.y);
    }
  };
  put_t(false);
  const float none = __int_as_float(0x7fffffff);
  const int c0 = 16 * warp;
  for (int col0 = 0; col0 < vdim; col0 += 128) {
    if (col0) {
      __syncthreads();
      load_values(col0);
    }
    spl_cp_wait<0>();
    __syncthreads();
    if (col0 + c0 < vdim) {
      float x[4][2][4] = {};
#pragma unroll
      for (int kt = 0; kt < DC / 16; ++kt) {
        uint32_t bv[2][2];
        spl_ldmatrix_x4_trans(bv[0][0], bv[0][1], bv[1][0], bv[1][1], v_s + (16 * kt + (lane & 15)) * LV + c0 + 8 * (lane >> 4));
#pragma unroll
        for (int m = kt; m < 4; ++m) {
          SplA a;
          spl_tri_a(a, tri, m, kt, lane);
          if (m == kt) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint32_t clean[1][2] = {{bv[i][0], bv[i][1]}};
              int first;
              const bool some = dc_take_out<1>(clean, first, t);
              spl_mma3_add<1>(reinterpret_cast<float(&)[1][4]>(x[m][i]), a, clean);
              if (some) dc_put_back(x[m][i], first, g, t);
            }
          } else {
            spl_mma3_add<2>(x[m], a, bv);
          }
        }
      }
      float* to = U + slot * DC * vdim + col0 + c0 + 2 * t;
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = 16 * m + 8 * e + g;
          const bool lost = i >= ok && i < n;
#pragma unroll
          for (int p = 0; p < 2; ++p)
            if (col0 + c0 + 8 * p + 2 * t < vdim)
              *reinterpret_cast<float2*>(to + (size_t)i * vdim + 8 * p) = lost ? make_float2(none, none) : make_float2(x[m][p][2 * e], x[m][p][2 * e + 1]);
        }
    }
  }
  __syncthreads();
  put_t(true);
  __syncthreads();
  float w[4][1][2][4] = {};
  if (c0 < DP) {
#pragma unroll
    for (int kt = 0; kt < DC / 16; ++kt) {
      SplB bk[2];
      const bf16* at = k_s + dc_at<DP>(16 * kt + (lane & 15), 2 * warp + (lane >> 4));
#pragma unroll
      for (int e = 0; e < 3; ++e) spl_ldmatrix_x4_trans(bk[0].p[e][0], bk[0].p[e][1], bk[1].p[e][0], bk[1].p[e][1], at + e * DC * DP);
#pragma unroll
      for (int m = kt; m < 4; ++m) {
        SplA a[1];
        spl_tri_a(a[0], tri, m, kt, lane);
        spl_mma6_add<1, 2>(w[m], a, bk);
      }
    }
  }
  __syncthreads();  // the keys are used up
  if (c0 < DP) {
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = 16 * m + 8 * e + g;
        const bool lost = i >= ok && i < n;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          uint32_t part[3];
          spl_pair(lost ? none : w[m][0][p][2 * e], lost ? none : w[m][0][p][2 * e + 1], part[0], part[1], part[2]);
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<uint32_t*>(k_s + q * DC * DP + dc_at<DP>(i, 2 * warp + p) + 2 * t) = part[q];
        }
      }
  }
  __syncthreads();
  uint4* to = reinterpret_cast<uint4*>(W + slot * 3 * DC * DP);
#pragma unroll 4
  for (int i = tid; i < 3 * DC * DP / 8; i += 256) to[i] = reinterpret_cast<const uint4*>(k_s)[i];
}

// ---------------------------------------------------------------- (2)
// 256 threads, one block an SM.  The state lies in the registers of its product's sums (a warp 16 rows), and, split into its parts, in shared
// memory for the next chunk's W S.  The parts of W and of the keys come chunk by chunk, each while the other is at work.  The serial chain of
// a chunk: 768 instructions of m16n8k16 in each of the two products of 32 columns, 3100 cycles of the tensor cores, and the splits and
// barriers between them: 7700 measured, 17 chunks of the longest sequence 80 us.
template <int DP, int COLS>
struct DcWalk {
  static constexpr int LS = COLS + 8;
  static constexpr int PARTS = 3 * DC * DP * 2;
  static constexpr int BYTES = 2 * PARTS + 3 * DP * LS * 2 + 3 * DC * LS * 2;
};
template <int DP, int COLS>
__global__ void __launch_bounds__(256)
delta_chunk_walk_kernel(const bf16* __restrict__ K, const float* __restrict__ tails, float* __restrict__ state, const int* __restrict__ slot_ids,
                        const int* __restrict__ seq_start, const bf16* __restrict__ W, float* __restrict__ U, float* __restrict__ states, int H,
                        int G, int dim, int vdim, int min_len, DcWindow win) {
  static_assert(DP == 128 || COLS == 32, "four warps to 16 rows each would share 16 columns");
  extern __shared__ __align__(16) unsigned char dc_smem[];
  using D = DcWalk<DP, COLS>;
  constexpr int LS = D::LS;
  constexpr int NA = COLS / 16;                 // pieces of eight columns that a warp has of W S ...
  constexpr int ROW_WARPS = DP / 16, NB = COLS / 8 * ROW_WARPS / 8;  // ... and of the state
  bf16* w_s = reinterpret_cast<bf16*>(dc_smem);                  // W's parts
  bf16* k_s = w_s + 3 * DC * DP;                                 // the keys'
  bf16* s_s = k_s + 3 * DC * DP;                                 // [3][DP][LS]
  bf16* u_s = s_s + 3 * DP * LS;                                 // [3][64][LS]: e^(L_63 - L_j) u_j
  __shared__ __align__(16) float tail[2][DC + 4];
  pdl_trigger();
  pdl_wait();
  const int col0 = blockIdx.x * COLS, h = blockIdx.y, s = blockIdx.z, kh = h / (H / G);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int start = __ldcg(seq_start + s), len = __ldcg(seq_start + s + 1) - start;
  const int n_chunks = win.count ? min((len + DC - 1) / DC, win.first + win.count) : (len + DC - 1) / DC;
  if (n_chunks <= win.first || len < min_len) return;
  auto load_w = [&](int c) {
    const size_t slot = (size_t)dc_chunk(win, start, s, c) * H + h;
    dc_load_parts<DP>(w_s, W + slot * 3 * DC * DP);
    if (tid < DC / 4 + 1) spl_cp16(&tail[c & 1][4 * tid], tails + slot * (DC + 4) + 4 * tid, true);
    spl_cp_commit();
  };
  load_w(win.first);
  // this lane's rows r0 + g and + 8 and its columns of the state; of W S: tokens m0 + g and + 8
  const int r0 = 16 * (warp % ROW_WARPS), sc = warp / ROW_WARPS * NB * 8, m0 = 16 * (warp & 3), uc = (warp >> 2) * NA * 8;
  float* record = state + ((size_t)__ldcg(slot_ids + s) * H + h) * dim * vdim + col0;
  float S[1][NB][4];
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    const int col = sc + 8 * i + 2 * t;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float2 v = make_float2(0.f, 0.f);
      if (r0 + g + 8 * e < dim && col0 + col < vdim) v = __ldcg(reinterpret_cast<const float2*>(record + (size_t)(r0 + g + 8 * e) * vdim + col));
      S[0][i][2 * e] = v.x, S[0][i][2 * e + 1] = v.y;
    }
  }
  for (int c = win.first; c < n_chunks; ++c) {
    const size_t chunk = dc_chunk(win, start, s, c), slot = chunk * H + h;
    // the chunk's X at this lane's places, asked for early
    float2 x[NA][2];
    float* u_at = U + (slot * DC + m0 + g) * vdim + col0 + uc + 2 * t;
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        x[i][e] = make_float2(0.f, 0.f);
        if (col0 + uc + 8 * i + 2 * t < vdim) x[i][e] = __ldcg(reinterpret_cast<const float2*>(u_at + (size_t)8 * e * vdim + 8 * i));
      }
    // the state before the chunk: for step (3), and in parts for W S
    float* keep = states + slot * dim * vdim + col0;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int col = sc + 8 * i + 2 * t;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = r0 + g + 8 * e;
        if (r < dim && col0 + col < vdim) *reinterpret_cast<float2*>(keep + (size_t)r * vdim + col) = make_float2(S[0][i][2 * e], S[0][i][2 * e + 1]);
        uint32_t part[3];
        spl_pair(S[0][i][2 * e], S[0][i][2 * e + 1], part[0], part[1], part[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(s_s + (p * DP + r) * LS + col) = part[p];
      }
    }
    spl_cp_wait<0>();
    __syncthreads();  // W and the state's parts are there; the keys are used up
    dc_load_parts<DP>(k_s, K + (chunk * G + kh) * 3 * DC * DP);
    spl_cp_commit();
    float acc[1][NA][4] = {};
#pragma unroll 2
    for (int kk = 0; kk < DP / 16; kk += 2) {
      SplB b[2][NA];
      if (NA == 2) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int p = 0; p < 3; ++p)
            spl_ldmatrix_x4_trans(b[j][0].p[p][0], b[j][0].p[p][1], b[j][NA - 1].p[p][0], b[j][NA - 1].p[p][1],
                                  s_s + (p * DP + 16 * (kk + j) + (lane & 15)) * LS + uc + 8 * (lane >> 4));
      } else {
#pragma unroll
        for (int p = 0; p < 3; ++p)
          spl_ldmatrix_x4_trans(b[0][0].p[p][0], b[0][0].p[p][1], b[1][0].p[p][0], b[1][0].p[p][1], s_s + (p * DP + 16 * kk + lane) * LS + uc);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        SplA a[1];
        dc_a<DP>(a[0], w_s, m0, kk + j, lane);
        spl_mma6_add<1, NA>(acc, a, b[j]);
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float f = tail[c & 1][m0 + g + 8 * e];
#pragma unroll
      for (int i = 0; i < NA; ++i) {
        const float2 u = make_float2(x[i][e].x - acc[0][i][2 * e], x[i][e].y - acc[0][i][2 * e + 1]);
        if (col0 + uc + 8 * i + 2 * t < vdim) *reinterpret_cast<float2*>(u_at + (size_t)8 * e * vdim + 8 * i) = u;
        uint32_t part[3];
        spl_pair(f * u.x, f * u.y, part[0], part[1], part[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(u_s + (p * DC + m0 + g + 8 * e) * LS + uc + 8 * i + 2 * t) = part[p];
      }
    }
    spl_cp_wait<0>();
    __syncthreads();  // the keys and U are there; W is used up
    if (c + 1 < n_chunks) load_w(c + 1);
    const float decay = tail[c & 1][DC];
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[0][i][e] *= decay;
#pragma unroll 2
    for (int kt = 0; kt < DC / 16; ++kt) {
      SplA a[1];
      SplB b[NB];
      const int p7 = lane & 7, mat = lane >> 3;
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        spl_ldmatrix_x4_trans(a[0].p[p][0], a[0].p[p][1], a[0].p[p][2], a[0].p[p][3],
                              k_s + p * DC * DP + dc_at<DP>(16 * kt + p7 + 8 * (mat >> 1), r0 / 8 + (mat & 1)));
#pragma unroll
        for (int i = 0; i < NB; i += 2)
          spl_ldmatrix_x4_trans(b[i].p[p][0], b[i].p[p][1], b[i + 1].p[p][0], b[i + 1].p[p][1],
                                u_s + (p * DC + 16 * kt + (lane & 15)) * LS + sc + 8 * i + 8 * (lane >> 4));
      }
      spl_mma6_add<1, NB>(S, a, b);
    }
  }
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    const int col = sc + 8 * i + 2 * t;
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (r0 + g + 8 * e < dim && col0 + col < vdim)
        *reinterpret_cast<float2*>(record + (size_t)(r0 + g + 8 * e) * vdim + col) = make_float2(S[0][i][2 * e], S[0][i][2 * e + 1]);
  }
}

// ---------------------------------------------------------------- (3)
// 256 threads, two blocks an SM, up to 128 values of a head (more: further blocks, which make the scores again).  A warp has all 64 tokens and
// 16 columns (eight in each half of the state's tile), so that U and the state, split as they are read, are split once.  Where the keys' parts
// were come the scores' and behind them the state, half by half, and U.
template <int DP>
struct DcOut {
  static constexpr int LU = 132, LS = 68;
  static constexpr int PARTS = 3 * DC * DP * 2, HALF = DP * LS * 4, VALUES = DC * LU * 4;
  static constexpr int LATER = 3 * SPL_TRI_BYTES + (HALF > VALUES ? HALF : VALUES);
  static constexpr int BYTES = PARTS + (PARTS > LATER ? PARTS : LATER);
};
template <int DP>
__global__ void __launch_bounds__(256, 2)
delta_chunk_out_kernel(const float* __restrict__ qn, const bf16* __restrict__ K, const float* __restrict__ log_decay,
                       const int* __restrict__ seq_start, const float* __restrict__ U, const float* __restrict__ states, void* __restrict__ out,
                       int out_stride, int H, int G, int dim, int vdim, int n_seqs, int min_len, DcWindow win, SplNorm norm) {
  extern __shared__ __align__(16) unsigned char dc_smem[];
  using D = DcOut<DP>;
  constexpr int LU = D::LU, LS = D::LS;
  bf16* q_s = reinterpret_cast<bf16*>(dc_smem);               // the queries' parts
  bf16* k_s = q_s + 3 * DC * DP;                              // the keys'
  unsigned char* p_s = dc_smem + D::PARTS;                    // the scores' parts
  float* s_s = reinterpret_cast<float*>(p_s + 3 * SPL_TRI_BYTES);  // [DP][LS]
  float* u_s = s_s;                                           // [64][LU]
  __shared__ double L[DC];
  pdl_trigger();
  pdl_wait();
  const int c = win.first + blockIdx.x, h = blockIdx.y, s = blockIdx.z % n_seqs, col0 = blockIdx.z / n_seqs * 128, kh = h / (H / G), tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int start = __ldcg(seq_start + s), end = __ldcg(seq_start + s + 1), t0 = start + c * DC;
  const int n = min(DC, end - t0);
  if (n <= 0 || end - start < min_len) return;
  const size_t chunk = dc_chunk(win, start, s, c), slot = chunk * H + h;
  {
    DcRows<DP> rows;
    rows.load(qn + ((size_t)t0 * G + kh) * dim, (size_t)G * dim, n, dim);
    dc_load_parts<DP>(k_s, K + (chunk * G + kh) * 3 * DC * DP);
    spl_cp_commit();
    if (tid < 32) dc_log_sums(log_decay, t0, n, H, h, L, tid);
#pragma unroll
    for (int p = 0; p < DcRows<DP>::PER; ++p) dc_put8<DP>(q_s, rows.row(p), rows.piece(p), rows.x[p], rows.y[p]);
  }
  spl_cp_wait<0>();
  __syncthreads();
  float inner[4][4];
  dc_inner_lower<DP>(inner, q_s, k_s, warp, lane);
  __syncthreads();  // the keys are used up
  dc_inner_each(inner, warp, lane, [&](int i, int j, float x, float y) {
    spl_tri_put(p_s, i, j, j <= i ? dc_decay(L[i], L[j]) * x : 0.f, j + 1 <= i ? dc_decay(L[i], L[j + 1]) * y : 0.f);
  });
  const float* sp = states + slot * dim * vdim + col0;
  float acc[2][2][2][1][4] = {};  // [half][32 tokens][16 of them]
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    if (half) __syncthreads();  // the first half is used up
#pragma unroll 4
    for (int idx = tid; idx < DP * 16; idx += 256) {  // columns 16 w + 8 half .. of every warp w
      const int r = idx >> 4, e = idx & 15, col = 16 * (e >> 1) + 8 * half + 4 * (e & 1);
      const bool here = r < dim && col0 + col < vdim;
      spl_cp16(s_s + r * LS + 4 * e, here ? sp + (size_t)r * vdim + col : states, here);
    }
    spl_cp_commit();
    spl_cp_wait<0>();
    __syncthreads();
    if (col0 + 16 * warp + 8 * half < vdim) {
#pragma unroll 1
      for (int kk = 0; kk < DP / 16; ++kk) {
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = s_s[(16 * kk + 2 * t + (e & 1) + 8 * (e >> 1)) * LS + 8 * warp + g];
        SplB b[1];
        spl_b(b[0], y);
#pragma unroll
        for (int mm = 0; mm < 2; ++mm) {
          SplA a[2];
#pragma unroll
          for (int m = 0; m < 2; ++m) dc_a<DP>(a[m], q_s, 16 * (2 * mm + m), kk, lane);
          spl_mma6_add<2, 1>(acc[half][mm], a, b);
        }
      }
    }
  }
  __syncthreads();  // the state is used up
#pragma unroll 4
  for (int i = tid; i < DC * 32; i += 256) {
    const int r = i >> 5, cc = (i & 31) * 4;
    const bool here = col0 + cc < vdim;
    spl_cp16(u_s + r * LU + cc, here ? U + (slot * DC + r) * vdim + col0 + cc : U, here);
  }
  spl_cp_commit();
#pragma unroll
  for (int m = 0; m < 4; ++m) {  // the decay since the chunk's start
    const float lo = dc_decay(L[16 * m + g], 0.0), hi = dc_decay(L[16 * m + g + 8], 0.0);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float(&y)[4] = acc[half][m >> 1][m & 1][0];
      y[0] *= lo, y[1] *= lo, y[2] *= hi, y[3] *= hi;
    }
  }
  spl_cp_wait<0>();
  __syncthreads();
#pragma unroll
  for (int kt = 0; kt < DC / 16; ++kt) {
    SplB b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = u_s[(16 * kt + 2 * t + (e & 1) + 8 * (e >> 1)) * LU + 16 * warp + 8 * i + g];
      spl_b(b[i], y);
    }
#pragma unroll
    for (int m = kt; m < 4; ++m) {
      SplA a[1];
      spl_tri_a(a[0], p_s, m, kt, lane);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float(&sum)[1][1][4] = reinterpret_cast<float(&)[1][1][4]>(acc[i][m >> 1][m & 1]);
        if (m == kt) {
          SplB clean[1] = {b[i]};
          int first;
          const bool some = dc_take_out<3>(clean[0].p, first, t);
          spl_mma6_add<1, 1>(sum, a, clean);
          if (some) dc_put_back(sum[0][0], first, g, t);
        } else {
          spl_mma6_add<1, 1>(sum, a, reinterpret_cast<const SplB(&)[1]>(b[i]));
        }
      }
    }
  }
  spl_finish(acc, reinterpret_cast<float*>(dc_smem), n, t0, h, vdim, col0, out, out_stride, norm);
}

// ---------------------------------------------------------------- host side
// Sizes these kernels are built for: key sizes in multiples of 4 up to 128, value sizes in multiples of 4.
RL_API int rl_delta_chunked_takes(int dim, int vdim) { return dim > 0 && vdim > 0 && dim <= 128 && dim % 4 == 0 && vdim % 4 == 0; }

// Floats of scratch for n_tokens tokens of n_seqs sequences: W's parts, the keys' parts, U, the states and the tails.
static long long chunk_floats(int H, int dim, int vdim) {
  return H * (2 * (3 * DC / 2) * (dim <= 64 ? 64LL : 128LL) + (long long)DC * vdim + (long long)dim * vdim + DC + 4);
}
RL_API long long rl_delta_chunked_scratch(int n_tokens, int n_seqs, int H, int dim, int vdim) {
  return ((long long)n_tokens / DC + n_seqs + 1) * chunk_floats(H, dim, vdim);
}
// How many chunks of every sequence a scratch of so many floats has room for at a time; 0: for all of them, -1: for none.
RL_API int rl_delta_chunked_window(long long scratch_floats, int n_tokens, int n_seqs, int H, int dim, int vdim) {
  if (n_seqs <= 0 || H <= 0 || dim <= 0 || vdim <= 0) return -1;
  if (scratch_floats >= rl_delta_chunked_scratch(n_tokens, n_seqs, H, dim, vdim)) return 0;
  const long long fit = scratch_floats / (n_seqs * chunk_floats(H, dim, vdim));
  return fit < 1 ? -1 : (int)(fit < 0x1000000 ? fit : 0x1000000);
}

// qn, kn: float32 [T, G dim] (unit vectors, the queries times their constant); v: bfloat16 rows of >= H vdim; beta, log_decay: float32
// [T, H]; state: float32 [slots, H, dim, vdim]; out: float32 [T, >= H vdim], or with norm_w (the heads' norm weights [vdim], up to 128
// values) bfloat16 rows that have been through what head_norm_gate does.  Sequences of fewer than min_len tokens (and their rows of out) are
// left alone.  window: 0, or how many chunks of every sequence to take at a time.
template <int DP>
static int launch_delta_chunked(const float* qn, const float* kn, const bf16* v, int v_stride, const float* beta, const float* log_decay,
                                float* state, const int* slot_ids, const int* seq_start, void* out, int out_stride, int n_tokens, int n_seqs,
                                int max_q_len, int H, int G, int dim, int vdim, int min_len, float* scratch, int window, const SplNorm& norm, cudaStream_t stream) {
  const long long chunks = window ? (long long)window * n_seqs : n_tokens / DC + n_seqs + 1;
  bf16* W = reinterpret_cast<bf16*>(scratch);
  bf16* K = W + chunks * H * 3 * DC * DP;
  float* U = reinterpret_cast<float*>(K + chunks * H * 3 * DC * DP);
  float* states = U + chunks * H * DC * vdim;
  float* tails = states + chunks * H * dim * vdim;  // [chunk][head][64 + 4]
  const int groups = (vdim + 127) / 128, all_chunks = (max_q_len + DC - 1) / DC, n_chunks = window && window < all_chunks ? window : all_chunks;
  if ((long long)groups * n_seqs > 65535) RL_REFUSE(4, "delta_chunked: %d sequences of %d values exceed the grid", n_seqs, vdim);
  const dim3 per_chunk(n_chunks, H, n_seqs), per_group(n_chunks, H, n_seqs * groups);
  const int v_wide = vdim % 8 == 0 && v_stride % 8 == 0 && ((uintptr_t)v & 15) == 0;
  // Blocks of 16 columns of the state, whose chain of chunks is shorter, where blocks of 32 would fill no more than two thirds of the SMs:
  // one prompt of 2048 tokens, 16 heads (64 blocks of 32): 89 us instead of 146; 700, 33 and 141 tokens, 8 heads (96): 32 instead of 49.
  // With more the second round of blocks costs what the chain gains: 1400 tokens, 32 heads (128): 122 instead of 106.
  const long long wide_blocks = (long long)((vdim + 31) / 32) * H * n_seqs;
  const bool narrow = DP == 128 && 3 * wide_blocks <= 2 * rl_sm_count();
  constexpr int s1 = DcSolve<DP>::BYTES, s3 = DcOut<DP>::BYTES;
  auto walk = DP == 128 && narrow ? delta_chunk_walk_kernel<128, 16> : delta_chunk_walk_kernel<DP, 32>;
  const int s2 = narrow ? DcWalk<128, 16>::BYTES : DcWalk<DP, 32>::BYTES, cols = narrow ? 16 : 32;
  if (cudaFuncSetAttribute(delta_chunk_solve_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, s1) != cudaSuccess ||
      cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, s2) != cudaSuccess ||
      cudaFuncSetAttribute(delta_chunk_out_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, s3) != cudaSuccess)
    RL_REFUSE(7, "delta_chunked: cannot get %d, %d or %d bytes of shared memory", s1, s2, s3);
  const dim3 per_tile((vdim + cols - 1) / cols, H, n_seqs);
  for (int first = 0; first < all_chunks; first += n_chunks) {
    const DcWindow win = {first, window};
    RL_LAUNCH_CHECK(rl_launch<false>(delta_chunk_solve_kernel<DP>, per_chunk, 256, s1, stream, kn, v, v_stride, v_wide, beta, log_decay, seq_start, W, K, U,
                                     tails, H, G, dim, vdim, min_len, win));
    RL_LAUNCH_CHECK(rl_launch(walk, per_tile, 256, s2, stream, (const bf16*)K, (const float*)tails, state, slot_ids, seq_start, (const bf16*)W, U, states,
                              H, G, dim, vdim, min_len, win));
    RL_LAUNCH_CHECK(rl_launch(delta_chunk_out_kernel<DP>, per_group, 256, s3, stream, qn, (const bf16*)K, log_decay, seq_start, (const float*)U,
                              (const float*)states, out, out_stride, H, G, dim, vdim, n_seqs, min_len, win, norm));
  }
  return 0;
}

RL_API int rl_delta_chunked(const float* qn, const float* kn, const void* v, int v_stride, const float* beta, const float* log_decay, float* state,
                            const int* slot_ids, const int* seq_start, void* out, int out_stride, int n_tokens, int n_seqs, int max_q_len, int H,
                            int G, int dim, int vdim, int min_len, float* scratch, long long scratch_floats, const float* norm_w, float eps, const void* gate, int gate_stride,
                            int gate_act, float out_scale, cudaStream_t stream) {
  if (n_tokens <= 0 || n_seqs <= 0 || max_q_len <= 0 || H <= 0 || G <= 0) RL_REFUSE(1, "delta_chunked: T=%d S=%d max_q=%d H=%d G=%d", n_tokens, n_seqs, max_q_len, H, G);
  if (!rl_delta_chunked_takes(dim, vdim)) RL_REFUSE(2, "delta_chunked: sizes %d / %d (multiples of 4, keys up to 128)", dim, vdim);
  if (H % G) RL_REFUSE(3, "delta_chunked: %d heads are not a multiple of %d q/k heads", H, G);
  if (H > 65535 || n_seqs > 65535) RL_REFUSE(4, "delta_chunked: %d heads or %d sequences exceed the grid", H, n_seqs);
  if (v_stride < H * vdim || out_stride < H * vdim) RL_REFUSE(5, "delta_chunked: rows of %d and %d for %d values", v_stride, out_stride, H * vdim);
  if (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)state | (uintptr_t)scratch) & 15) RL_REFUSE(6, "delta_chunked: operands must be 16-byte aligned");
  if (!norm_w && (out_stride % 4 || ((uintptr_t)out & 15))) RL_REFUSE(6, "delta_chunked: the result's rows must be 16-byte aligned");
  // (rows of whole fours: a step with sequences of a few tokens has the norm made by head_norm_gate, four columns a lane, and the bits are the same)
  if (norm_w && (vdim > 128 || out_stride % 4 || ((uintptr_t)out & 7) || gate_stride % 4 || ((uintptr_t)gate & 7) || ((uintptr_t)norm_w & 7)))
    return RL_NOT_FUSED;
  const int window = rl_delta_chunked_window(scratch_floats, n_tokens, n_seqs, H, dim, vdim);
  if (window < 0) RL_REFUSE(8, "delta_chunked: %lld floats of scratch hold no chunk of %d sequences", scratch_floats, n_seqs);
  const SplNorm norm{norm_w, eps, (const bf16*)gate, gate_stride, gate_act, out_scale};
  if (dim <= 64)
    return launch_delta_chunked<64>(qn, kn, (const bf16*)v, v_stride, beta, log_decay, state, slot_ids, seq_start, out, out_stride, n_tokens, n_seqs,
                                    max_q_len, H, G, dim, vdim, min_len, scratch, window, norm, stream);
  return launch_delta_chunked<128>(qn, kn, (const bf16*)v, v_stride, beta, log_decay, state, slot_ids, seq_start, out, out_stride, n_tokens, n_seqs,
                                   max_q_len, H, G, dim, vdim, min_len, scratch, window, norm, stream);
}
