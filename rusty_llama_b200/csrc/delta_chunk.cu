// The gated delta rule for prompts of a bfloat16 run, chunk by chunk instead of token by token (delta_rule.cu has the rule and the
// token-by-token kernel, which takes single tokens, short portions and 32-bit runs).  All arithmetic is 32-bit FMA, as there.
//
// Inside a chunk of 64 tokens, with L_i the sum of the log decays up to token i and S_0 the state before the chunk,
//
//     S_i = e^(L_i) S_0 + sum_(j <= i) e^(L_i - L_j) k_j u_j^T,      u_i = beta_i (v_i - e^(L_i) S_0^T k_i - sum_(j < i) e^(L_i - L_j) (k_i . k_j) u_j)
//
// so the u of a chunk solve a unit triangular system (I + A) U = diag(beta) (V - diag(e^L) K S_0), A_ij = beta_i e^(L_i - L_j) (k_i . k_j)
// for j < i, and with  (I + A) [X | W] = [diag(beta) V | diag(beta e^L) K]  they are U = X - W S_0.  Decays only enter as e to the
// difference of two sums where the difference is not positive: nothing overflows, what underflows is zero.
//
//   (1) delta_chunk_solve   per (chunk, head): A, then X and W by forward substitution, a thread a column of 64 registers
//   (2) delta_chunk_walk    per (32 columns of the state, head, sequence), chunk after chunk: U = X - W S, S <- e^(L_63) S + K^T (e^(L_63 - L) U);
//                           leaves U in X's place and the state before every chunk
//   (3) delta_chunk_out     per (chunk, head): O = diag(e^L) Q S_0 + (Q K^T * e^(L_i - L_j), j <= i) U
//
// Token by token every token was one chain of dependent steps per column (760 cycles with nothing to hide them); here only (2) is
// serial, with 64 tokens a step.  Bound: the FMA pipe and the shared-memory reads that feed it, 1.1 billion multiply-adds for 16 heads
// of 128 x 128 and 2048 tokens in (2) and about as many in (1) and (3) each.  Sequences of 1029, 700 and 319 tokens: 62, 106 and 72 us
// against 444 us token by token.
#include "common.cuh"

RL_DEFINE_ERROR_TEXT()

#define DC 64          // tokens per chunk
#define DC_COLS 32     // columns of the state that a block of (2) walks with
#define DC_OUT_COLS 64 // columns of the output that (3) does at a time
#define DC_PAD 4       // floats between rows in shared memory: neighbouring rows start four banks apart

// Chunks are numbered over the whole call: those of sequence s start at seq_start[s] / 64 + s (room for every sequence's last, partly
// filled one).
__device__ __forceinline__ int dc_first_chunk(int start, int s) { return start / DC + s; }

__device__ __forceinline__ void dc_cp_async16(float* dst, const float* src, bool here) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(here ? 16 : 0) : "memory");
}

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

// 64 rows of dim numbers, `ld` apart, on their way into shared memory [64][DP + DC_PAD]; rows from n on and columns from dim on are
// zeros.  (All copies of a tile are asked for before any is waited for: loaded piece by piece, the tiles' latencies took most of the time.)
template <int DP, int THREADS>
__device__ __forceinline__ void dc_load_rows(float* dst, const float* __restrict__ src, size_t ld, int n, int dim) {
  constexpr int Q = DP / 4;
#pragma unroll 4
  for (int i = threadIdx.x; i < DC * Q; i += THREADS) {
    const int r = i / Q, k = (i % Q) * 4;
    const bool here = r < n && k < dim;
    dc_cp_async16(dst + r * (DP + DC_PAD) + k, here ? src + r * ld + k : src, here);
  }
}
__device__ __forceinline__ void dc_landed() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// acc[a][b] += sum_k x[ty + 16 a][k] * y[tx + 16 b][k]: 64 x 64 inner products of rows by 256 threads
template <int DP>
__device__ __forceinline__ void dc_inner(const float* x, const float* y, int ty, int tx, float (&acc)[4][4]) {
  constexpr int LD = DP + DC_PAD;
#pragma unroll 4
  for (int k = 0; k < DP; k += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = *reinterpret_cast<const float4*>(x + (ty + 16 * i) * LD + k);
      b[i] = *reinterpret_cast<const float4*>(y + (tx + 16 * i) * LD + k);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
        acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
        acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
      }
  }
}

// ---------------------------------------------------------------- (1)
template <int DP>
__global__ void __launch_bounds__(256, 2)
delta_chunk_solve_kernel(const float* __restrict__ kn, const bf16* __restrict__ v, int v_stride, const float* __restrict__ beta,
                         const float* __restrict__ log_decay, const int* __restrict__ seq_start, float* __restrict__ W, float* __restrict__ U,
                         float* __restrict__ tails, int H, int G, int dim, int vdim, int min_len) {
  extern __shared__ __align__(16) float sm[];
  constexpr int LD = DP + DC_PAD, LA = DC + DC_PAD;
  float* k_s = sm;             // [64][LD]
  float* a_s = k_s + DC * LD;  // [64][LA]: A transposed, a_s[j][i] = A_ij
  __shared__ double L[DC];
  __shared__ float be[DC], from_start[DC];
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x, h = blockIdx.y, s = blockIdx.z, kh = h / (H / G), tid = threadIdx.x;
  const int start = __ldcg(seq_start + s), end = __ldcg(seq_start + s + 1), t0 = start + c * DC;
  const int n = min(DC, end - t0);
  if (n <= 0 || end - start < min_len) return;
  dc_load_rows<DP, 256>(k_s, kn + ((size_t)t0 * G + kh) * dim, (size_t)G * dim, n, dim);
  if (tid < 32) dc_log_sums(log_decay, t0, n, H, h, L, tid);
  if (tid >= 64 && tid < 64 + DC) be[tid - 64] = tid - 64 < n ? __ldcg(beta + (size_t)(t0 + tid - 64) * H + h) : 0.f;
  dc_landed();
  {
    const int ty = tid >> 4, tx = tid & 15;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    dc_inner<DP>(k_s, k_s, ty, tx, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int i = tx + 16 * b, j = ty + 16 * a;  // (symmetric: the thread's columns serve as i, so that neighbours write side by side)
        a_s[j * LA + i] = j < i ? be[i] * dc_decay(L[i], L[j]) * acc[a][b] : 0.f;
      }
  }
  const size_t row0 = ((size_t)(dc_first_chunk(start, s) + c) * H + h) * DC;
  if (tid < DC) from_start[tid] = dc_decay(L[tid], 0.0);
  __syncthreads();
  if (tid < DC) {  // what is left of a token's write, and of the state before the chunk, at the chunk's end
    tails[row0 / DC * (DC + 4) + tid] = dc_decay(L[DC - 1], L[tid]);
    if (tid == 0) tails[row0 / DC * (DC + 4) + DC] = dc_decay(L[DC - 1], 0.0);
  }
  for (int col = tid; col < dim + vdim; col += 256) {
    float R[DC];
    if (col < dim) {
#pragma unroll
      for (int i = 0; i < DC; ++i) R[i] = be[i] * from_start[i] * k_s[i * LD + col];
    } else {
      const bf16* vc = v + (size_t)t0 * v_stride + (size_t)h * vdim + (col - dim);
#pragma unroll
      for (int i = 0; i < DC; ++i) R[i] = i < n ? be[i] * __bfloat162float(vc[(size_t)i * v_stride]) : 0.f;
    }
    // row j is final once the rows before it have been taken out of it; then it is taken out of the later ones (independent sums)
#pragma unroll
    for (int j = 0; j < DC - 1; ++j) {
      const float x = -R[j];
      asm volatile("" ::: "memory");  // (no further ahead with the loads: they would push the column out of the registers)
#pragma unroll
      for (int i = (j + 1) & ~3; i < DC; i += 4) {
        const float4 a = *reinterpret_cast<const float4*>(a_s + j * LA + i);
        if (i > j) R[i] = fmaf(a.x, x, R[i]);
        if (i + 1 > j) R[i + 1] = fmaf(a.y, x, R[i + 1]);
        if (i + 2 > j) R[i + 2] = fmaf(a.z, x, R[i + 2]);
        if (i + 3 > j) R[i + 3] = fmaf(a.w, x, R[i + 3]);
      }
    }
    float* to = col < dim ? W + row0 * dim + col : U + row0 * vdim + (col - dim);
    const int ld = col < dim ? dim : vdim;
#pragma unroll
    for (int i = 0; i < DC; ++i) to[(size_t)i * ld] = R[i];
  }
}

// ---------------------------------------------------------------- (2)
// A block of 4 DP threads: a warp has 16 rows of 16 of its columns of the state, a lane 4 x 2 of them in registers.  (Blocks of 16 columns
// with one warp a sub-core left its latencies open, with two they still did:
// 130 and 123 us, now 106, for sequences of 1029, 700 and 319 tokens and 16 heads of 128.  One of 2048 takes 191: 6 us a chunk.)
template <int DP>
__global__ void __launch_bounds__(4 * DP)
delta_chunk_walk_kernel(const float* __restrict__ kn, const float* __restrict__ tails, float* __restrict__ state,
                        const int* __restrict__ slot_ids, const int* __restrict__ seq_start, const float* __restrict__ W, float* __restrict__ U,
                        float* __restrict__ states, int H, int G, int dim, int vdim, int min_len) {
  extern __shared__ __align__(16) float sm[];
  constexpr int LD = DP + DC_PAD, PARTS = DP / 32, LS = DC_COLS + DC_PAD, THREADS = 4 * DP;
  float* w_s = sm;                      // [2][64][LD]
  float* k_s = w_s + 2 * DC * LD;       // [2][64][LD]
  float* s_s = k_s + 2 * DC * LD;       // [DP][LS]: the state before the chunk
  float* u_s = s_s + DP * LS;           // [64][32]: e^(L_63 - L_j) u_j
  float* part = u_s + DC * DC_COLS;     // [PARTS][64][32]
  __shared__ __align__(16) float tail[2][DC + 4];
  pdl_trigger();
  pdl_wait();
  const int col0 = blockIdx.x * DC_COLS, h = blockIdx.y, s = blockIdx.z, kh = h / (H / G);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int start = __ldcg(seq_start + s), len = __ldcg(seq_start + s + 1) - start, n_chunks = (len + DC - 1) / DC;
  if (n_chunks <= 0 || len < min_len) return;
  const int chunk0 = dc_first_chunk(start, s);
  auto load = [&](int c) {
    const size_t slot = (size_t)(chunk0 + c) * H + h;
    dc_load_rows<DP, THREADS>(w_s + (c & 1) * DC * LD, W + slot * DC * dim, dim, DC, dim);
    dc_load_rows<DP, THREADS>(k_s + (c & 1) * DC * LD, kn + ((size_t)(start + c * DC) * G + kh) * dim, (size_t)G * dim, min(DC, len - c * DC), dim);
    if (tid < DC / 4 + 1) dc_cp_async16(&tail[c & 1][4 * tid], tails + slot * (DC + 4) + 4 * tid, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0);
  const int column_half = 16 * (warp / (DP / 16)), row_warp = warp % (DP / 16);
  const int kg = 16 * row_warp + (lane >> 3) * 4, c2 = column_half + (lane & 7) * 2;  // this lane's 4 rows and 2 columns of the state
  const bool cols_here = col0 + c2 < vdim;                          // (vdim is a multiple of 4)
  float* record = state + ((size_t)__ldcg(slot_ids + s) * H + h) * dim * vdim + col0 + c2;
  float2 S[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    S[e] = make_float2(0.f, 0.f);
    if (cols_here && kg + e < dim) S[e] = __ldcg(reinterpret_cast<const float2*>(record + (size_t)(kg + e) * vdim));
  }
  for (int c = 0; c < n_chunks; ++c) {
    const size_t slot = (size_t)(chunk0 + c) * H + h;
    // the chunk's X at this thread's places of the sum below, asked for early
    constexpr int PER = DC * DC_COLS / 4 / THREADS;
    float x[PER][4];
    float* u_at[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int i = tid + p * THREADS, row = i / (DC_COLS / 4), cc = i % (DC_COLS / 4) * 4;
      u_at[p] = U + (slot * DC + row) * vdim + col0 + cc;
      x[p][0] = x[p][1] = x[p][2] = x[p][3] = 0.f;
      if (col0 + cc < vdim) load4_g(u_at[p], x[p]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      *reinterpret_cast<float2*>(s_s + (kg + e) * LS + c2) = S[e];
      if (cols_here && kg + e < dim) *reinterpret_cast<float2*>(states + (slot * dim + kg + e) * vdim + col0 + c2) = S[e];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the chunk's rows and the state are there; everyone is done with the chunk before
    if (c + 1 < n_chunks) load(c + 1);
    const float* w = w_s + (c & 1) * DC * LD, *k = k_s + (c & 1) * DC * LD;
    {  // W S: this warp takes 32 rows of S and half of the tokens: (lane / 4) + 8 i of them, four columns
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
      const int kw = row_warp % PARTS, rg = (lane >> 2) + 32 * (row_warp / PARTS), cg = column_half + (lane & 3) * 4;
#pragma unroll 4
      for (int kk = 32 * kw; kk < 32 * kw + 32; kk += 4) {
        float4 sv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) sv[e] = *reinterpret_cast<const float4*>(s_s + (kk + e) * LS + cg);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(w + (rg + 8 * i) * LD + kk);
          acc[i][0] = fmaf(a.x, sv[0].x, acc[i][0]); acc[i][1] = fmaf(a.x, sv[0].y, acc[i][1]); acc[i][2] = fmaf(a.x, sv[0].z, acc[i][2]); acc[i][3] = fmaf(a.x, sv[0].w, acc[i][3]);
          acc[i][0] = fmaf(a.y, sv[1].x, acc[i][0]); acc[i][1] = fmaf(a.y, sv[1].y, acc[i][1]); acc[i][2] = fmaf(a.y, sv[1].z, acc[i][2]); acc[i][3] = fmaf(a.y, sv[1].w, acc[i][3]);
          acc[i][0] = fmaf(a.z, sv[2].x, acc[i][0]); acc[i][1] = fmaf(a.z, sv[2].y, acc[i][1]); acc[i][2] = fmaf(a.z, sv[2].z, acc[i][2]); acc[i][3] = fmaf(a.z, sv[2].w, acc[i][3]);
          acc[i][0] = fmaf(a.w, sv[3].x, acc[i][0]); acc[i][1] = fmaf(a.w, sv[3].y, acc[i][1]); acc[i][2] = fmaf(a.w, sv[3].z, acc[i][2]); acc[i][3] = fmaf(a.w, sv[3].w, acc[i][3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) store4(part + (kw * DC + rg + 8 * i) * DC_COLS + cg, acc[i]);
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int i = tid + p * THREADS, row = i / (DC_COLS / 4), cc = i % (DC_COLS / 4) * 4;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ww = 0; ww < PARTS; ++ww) {
        float y[4];
        load4(part + (ww * DC + row) * DC_COLS + cc, y);
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] += y[e];
      }
      const float f = tail[c & 1][row];
      float scaled[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[p][e] -= sum[e];
        scaled[e] = f * x[p][e];
      }
      if (col0 + cc < vdim) store4(u_at[p], x[p]);
      store4(u_s + row * DC_COLS + cc, scaled);
    }
    __syncthreads();
    const float g = tail[c & 1][DC];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      S[e].x *= g;
      S[e].y *= g;
    }
#pragma unroll 8
    for (int j = 0; j < DC; ++j) {
      const float4 a = *reinterpret_cast<const float4*>(k + j * LD + kg);
      const float2 b = *reinterpret_cast<const float2*>(u_s + j * DC_COLS + c2);
      S[0].x = fmaf(a.x, b.x, S[0].x); S[0].y = fmaf(a.x, b.y, S[0].y);
      S[1].x = fmaf(a.y, b.x, S[1].x); S[1].y = fmaf(a.y, b.y, S[1].y);
      S[2].x = fmaf(a.z, b.x, S[2].x); S[2].y = fmaf(a.z, b.y, S[2].y);
      S[3].x = fmaf(a.w, b.x, S[3].x); S[3].y = fmaf(a.w, b.y, S[3].y);
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (cols_here && kg + e < dim) *reinterpret_cast<float2*>(record + (size_t)(kg + e) * vdim) = S[e];
}

// ---------------------------------------------------------------- (3)
// acc[a][e] += sum_k x[ty + 16 a][k] * y[k][4 tx + e]
template <int KN, int LX>
__device__ __forceinline__ void dc_outer(const float* x, const float* y, int ty, int tx, float (&acc)[4][4]) {
  constexpr int LY = DC_OUT_COLS + DC_PAD;
#pragma unroll 4
  for (int k = 0; k < KN; k += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = *reinterpret_cast<const float4*>(x + (ty + 16 * i) * LX + k);
      b[i] = *reinterpret_cast<const float4*>(y + (k + i) * LY + 4 * tx);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][0] = fmaf(av[j], b[j].x, acc[i][0]);
        acc[i][1] = fmaf(av[j], b[j].y, acc[i][1]);
        acc[i][2] = fmaf(av[j], b[j].z, acc[i][2]);
        acc[i][3] = fmaf(av[j], b[j].w, acc[i][3]);
      }
    }
  }
}

// The same over the tokens up to each row's own, acc[a][e] += sum_(k <= row) x[row][k] * y[k][4 tx + e], row = ty + 16 a.  What a row does not
// see is left out and not multiplied by zero: a later token's write may be infinite or no number.
template <int LX>
__device__ __forceinline__ void dc_outer_seen(const float* x, const float* y, int ty, int tx, float (&acc)[4][4]) {
  constexpr int LY = DC_OUT_COLS + DC_PAD;
#pragma unroll
  for (int sub = 0; sub < 4; ++sub) {
#pragma unroll 2
    for (int k = 0; k < 16; k += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(y + (16 * sub + k + j) * LY + 4 * tx);
#pragma unroll
      for (int i = sub; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(x + (ty + 16 * i) * LX + 16 * sub + k);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i > sub || k + j <= ty) {
            acc[i][0] = fmaf(av[j], b[j].x, acc[i][0]);
            acc[i][1] = fmaf(av[j], b[j].y, acc[i][1]);
            acc[i][2] = fmaf(av[j], b[j].z, acc[i][2]);
            acc[i][3] = fmaf(av[j], b[j].w, acc[i][3]);
          }
      }
    }
  }
}

template <int DP>
__global__ void __launch_bounds__(256, 2)
delta_chunk_out_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ log_decay,
                       const int* __restrict__ seq_start, const float* __restrict__ U, const float* __restrict__ states, float* __restrict__ out,
                       int out_stride, int H, int G, int dim, int vdim, int min_len) {
  extern __shared__ __align__(16) float sm[];
  constexpr int LD = DP + DC_PAD, LP = DC + DC_PAD, LY = DC_OUT_COLS + DC_PAD;
  constexpr int K_FLOATS = DC * LD > DP * LY ? DC * LD : DP * LY;
  float* q_s = sm;                // [64][LD]
  float* k_s = q_s + DC * LD;     // [64][LD]; then the state's tile [DP][LY]
  float* p_s = k_s + K_FLOATS;    // [64][LP]
  float* u_s = p_s + DC * LP;     // [64][LY]
  __shared__ double L[DC];
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x, h = blockIdx.y, s = blockIdx.z, kh = h / (H / G), tid = threadIdx.x;
  const int start = __ldcg(seq_start + s), end = __ldcg(seq_start + s + 1), t0 = start + c * DC;
  const int n = min(DC, end - t0);
  if (n <= 0 || end - start < min_len) return;
  const size_t at = ((size_t)t0 * G + kh) * dim, ld = (size_t)G * dim;
  dc_load_rows<DP, 256>(q_s, qn + at, ld, n, dim);
  dc_load_rows<DP, 256>(k_s, kn + at, ld, n, dim);
  if (tid < 32) dc_log_sums(log_decay, t0, n, H, h, L, tid);
  dc_landed();
  const int ty = tid >> 4, tx = tid & 15;
  {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    dc_inner<DP>(q_s, k_s, ty, tx, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        p_s[i * LP + j] = j <= i ? dc_decay(L[i], L[j]) * acc[a][b] : 0.f;
      }
  }
  const size_t slot = (size_t)(dc_first_chunk(start, s) + c) * H + h;
  for (int col0 = 0; col0 < vdim; col0 += DC_OUT_COLS) {
    __syncthreads();  // the keys (or the tile before) are used up
#pragma unroll 4
    for (int i = tid; i < (DP + DC) * (DC_OUT_COLS / 4); i += 256) {
      const int r = i / (DC_OUT_COLS / 4), cc = i % (DC_OUT_COLS / 4) * 4;
      const bool of_state = r < DP, here = col0 + cc < vdim && (!of_state || r < dim);
      const float* src = of_state ? states + (slot * dim + r) * vdim : U + (slot * DC + r - DP) * vdim;
      dc_cp_async16((of_state ? k_s + r * LY : u_s + (r - DP) * LY) + cc, here ? src + col0 + cc : states, here);
    }
    dc_landed();
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    dc_outer<DP, LD>(q_s, k_s, ty, tx, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const float f = dc_decay(L[ty + 16 * a], 0.0);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[a][e] *= f;
    }
    dc_outer_seen<LP>(p_s, u_s, ty, tx, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = ty + 16 * a;
      if (i < n && col0 + 4 * tx < vdim) store4(out + (size_t)(t0 + i) * out_stride + (size_t)h * vdim + col0 + 4 * tx, acc[a]);
    }
  }
}

// ---------------------------------------------------------------- host side
// Sizes these kernels are built for: key sizes in multiples of 4 up to 128, value sizes in multiples of 4.
RL_API int rl_delta_chunked_takes(int dim, int vdim) { return dim > 0 && vdim > 0 && dim <= 128 && dim % 4 == 0 && vdim % 4 == 0; }

// Floats of scratch for n_tokens tokens of n_seqs sequences.
RL_API long long rl_delta_chunked_scratch(int n_tokens, int n_seqs, int H, int dim, int vdim) {
  const long long chunks = n_tokens / DC + n_seqs + 1;
  return chunks * H * ((long long)DC * (dim + vdim) + (long long)dim * vdim + DC + 4);
}

// qn, kn: float32 [T, G dim] (unit vectors, the queries times their constant); v: bfloat16 rows of >= H vdim; beta, log_decay: float32
// [T, H]; state: float32 [slots, H, dim, vdim]; out: float32 [T, >= H vdim].  Sequences of fewer than min_len tokens (and their rows of out)
// are left alone.
template <int DP>
static int launch_delta_chunked(const float* qn, const float* kn, const bf16* v, int v_stride, const float* beta, const float* log_decay,
                                float* state, const int* slot_ids, const int* seq_start, float* out, int out_stride, int n_tokens, int n_seqs,
                                int max_q_len, int H, int G, int dim, int vdim, int min_len, float* scratch, cudaStream_t stream) {
  constexpr int LD = DP + DC_PAD, LY = DC_OUT_COLS + DC_PAD;
  constexpr size_t smem1 = (size_t)(DC * LD + DC * (DC + DC_PAD)) * 4;
  constexpr size_t smem2 = (size_t)(4 * DC * LD + DP * (DC_COLS + DC_PAD) + DC * DC_COLS + DP / 32 * DC * DC_COLS) * 4;
  constexpr size_t smem3 = (size_t)(DC * LD + (DC * LD > DP * LY ? DC * LD : DP * LY) + DC * (DC + DC_PAD) + DC * LY) * 4;
  if (cudaFuncSetAttribute(delta_chunk_solve_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1) != cudaSuccess ||
      cudaFuncSetAttribute(delta_chunk_walk_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2) != cudaSuccess ||
      cudaFuncSetAttribute(delta_chunk_out_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem3) != cudaSuccess)
    RL_REFUSE(7, "delta_chunked: cannot get %zu, %zu or %zu bytes of shared memory", smem1, smem2, smem3);
  const long long chunks = n_tokens / DC + n_seqs + 1;
  float* W = scratch;
  float* U = W + chunks * H * DC * dim;
  float* states = U + chunks * H * DC * vdim;
  float* tails = states + chunks * H * dim * vdim;  // [chunk][head][64 + 4]
  const dim3 per_chunk((max_q_len + DC - 1) / DC, H, n_seqs), per_tile((vdim + DC_COLS - 1) / DC_COLS, H, n_seqs);
  RL_LAUNCH_CHECK(rl_launch<false>(delta_chunk_solve_kernel<DP>, per_chunk, 256, smem1, stream, kn, v, v_stride, beta, log_decay, seq_start, W, U, tails, H, G, dim, vdim, min_len));
  RL_LAUNCH_CHECK(rl_launch(delta_chunk_walk_kernel<DP>, per_tile, 4 * DP, smem2, stream, kn, (const float*)tails, state, slot_ids, seq_start, (const float*)W, U, states,
                            H, G, dim, vdim, min_len));
  RL_LAUNCH_CHECK(rl_launch(delta_chunk_out_kernel<DP>, per_chunk, 256, smem3, stream, qn, kn, log_decay, seq_start, (const float*)U,
                            (const float*)states, out, out_stride, H, G, dim, vdim, min_len));
  return 0;
}

RL_API int rl_delta_chunked(const float* qn, const float* kn, const void* v, int v_stride, const float* beta, const float* log_decay, float* state,
                            const int* slot_ids, const int* seq_start, float* out, int out_stride, int n_tokens, int n_seqs, int max_q_len, int H,
                            int G, int dim, int vdim, int min_len, float* scratch, cudaStream_t stream) {
  if (n_tokens <= 0 || n_seqs <= 0 || max_q_len <= 0 || H <= 0 || G <= 0) RL_REFUSE(1, "delta_chunked: T=%d S=%d max_q=%d H=%d G=%d", n_tokens, n_seqs, max_q_len, H, G);
  if (!rl_delta_chunked_takes(dim, vdim)) RL_REFUSE(2, "delta_chunked: sizes %d / %d (multiples of 4, keys up to 128)", dim, vdim);
  if (H % G) RL_REFUSE(3, "delta_chunked: %d heads are not a multiple of %d q/k heads", H, G);
  if (H > 65535 || n_seqs > 65535) RL_REFUSE(4, "delta_chunked: %d heads or %d sequences exceed the grid", H, n_seqs);
  if (v_stride < H * vdim || out_stride < H * vdim || out_stride % 4) RL_REFUSE(5, "delta_chunked: rows of %d and %d for %d values", v_stride, out_stride, H * vdim);
  if (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)state | (uintptr_t)out | (uintptr_t)scratch) & 15) RL_REFUSE(6, "delta_chunked: operands must be 16-byte aligned");
  if (dim <= 64)
    return launch_delta_chunked<64>(qn, kn, (const bf16*)v, v_stride, beta, log_decay, state, slot_ids, seq_start, out, out_stride, n_tokens, n_seqs,
                                    max_q_len, H, G, dim, vdim, min_len, scratch, stream);
  return launch_delta_chunked<128>(qn, kn, (const bf16*)v, v_stride, beta, log_decay, state, slot_ids, seq_start, out, out_stride, n_tokens, n_seqs,
                                   max_q_len, H, G, dim, vdim, min_len, scratch, stream);
}
