// The matrix products of the true 32-bit path: out[M, N] = x[M, K] . w[N, K]^T
// with 32-bit inputs, FMA on the CUDA cores and no tensor-core instruction, so
// nothing is rounded to a shorter type on the way (the reference's oracle is its
// CPU backend, a 32-bit dot product per output: src/backend/cpu.rs:107-136).
//
// The order of every output's sum is fixed: k is cut into consecutive chunks of
// KCHUNK, counted from 0; a chunk is one running sum in ascending order, started
// at zero; the chunks' sums are added up in ascending order.  It depends neither
// on M nor on where the element lies in its tile nor on which of the two kernels
// below runs.  A row's result is therefore the same bits whether it is computed
// alone, inside a prompt or inside a batch.
//
// Why chunks: with one running sum over all of k, a product with few rows had a
// chain of K dependent FMAs per output and one thread for it (N / 64 blocks of a
// tile kernel: 32 of them for the 2048 features of an output projection).  A chunk
// per thread gives K / 128 times the threads and chains of 128.
//
//   gemv_f32_kernel  up to GEMV_ROWS rows: bound by reading the weights.  One row of 11264 x 2048: 18.6 us, 5.0 TB/s; 2048 x 5632: 11.9 us, 3.9 TB/s.
//   gemm_f32_kernel  more rows, and operands that cannot be moved 16 bytes at a time: bound by the FMA pipe.  283 rows of
//                    11264 x 2048: 344 us, 38 TFLOP/s; of 2048 x 2048, where the tiles are few: 84 us, 28 TFLOP/s.
// Prompts of 219 and 64 tokens and twelve decode steps of both on three layers of d 2048 and ff 5632: 60.9 ms in one kernel that
// held 64 x 64 tiles in registers whatever the rows, 6.1 ms in these two.
//
// gemm_fma_kernel with bfloat16 operands (widened on load, 32-bit sums over k in ascending order, the
// result rounded once, optionally through silu(gate) * up of neighbouring columns) takes the bfloat16
// products whose k is no multiple of 8: the streaming and tensor-core kernels move rows in 16-byte pieces and refuse
// those.  It is slow and only there so that every size a configuration allows runs.
#include "common.cuh"

RL_DEFINE_ERROR_TEXT()

#define TM 64
#define TN 64
#define TK 16

// SWIGLU: w's rows alternate gate and up; out[M, N/2] = gated_act(gate, up) from the 32-bit sums (silu(gate) * up,
// or the form with limits: see common.cuh).
template <typename TA, typename TO, bool SWIGLU>
__global__ void __launch_bounds__(256)
gemm_fma_kernel(const TA* __restrict__ x, int ldx, const TA* __restrict__ w, int ldw,
                TO* __restrict__ out, int ldo, int M, int N, int K, float act_alpha, float act_limit) {
  __shared__ float xs[TK][TM + 4];
  __shared__ float ws[TK][TN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  const int ty = tid / 16, tx = tid % 16;  // 16 x 16 threads, 4 x 4 outputs each
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += TK) {
    // 64 rows x 16 k of each operand: 1024 values, 4 per thread
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256;
      const int r = idx / TK, c = idx % TK;
      const int k = k0 + c;
      xs[c][r] = (m0 + r < M && k < K) ? to_f32(x[(size_t)(m0 + r) * ldx + k]) : 0.f;
      ws[c][r] = (n0 + r < N && k < K) ? to_f32(w[(size_t)(n0 + r) * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < TK; ++c) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[c][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[c][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
    if (SWIGLU) {
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const int n = n0 + tx * 4 + j;  // even: the gate's row; n + 1: the up's
        if (n + 1 < N) out[(size_t)m * ldo + n / 2] = from_f32<TO>(gated_act(acc[i][j], acc[i][j + 1], act_alpha, act_limit));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + tx * 4 + j;
        if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(acc[i][j]);
      }
    }
  }
}

// ------------------------------------------------------------------ 32-bit, few rows
#define KCHUNK 128        // the summation order's chunk of k: part of the result, not a tuning knob
#define GEMV_ROWS 8       // rows up to which the weights are streamed (measured, gate/up of 11264 x 2048: 8 rows 43 us; 17 rows in tiles 71 us)
#define GEMV_THREADS 128  // one (feature, chunk) pair each
#define GEMV_SUB 32       // k of a chunk that a stage of the ring holds: 128 bytes of an item, whose 16-byte pieces lie swizzled by the item
#define GEMV_XCHUNK (KCHUNK + 4)      // the rows of x, per chunk: eight chunks' same places meet all banks
#define GEMV_MAX_ITEMS 2048           // items of a block, whose sums wait in shared memory
#define GEMV_FEW 8                    // features that make up for what a block reads of x
#define GEMV_STAGE_BYTES (GEMV_THREADS * GEMV_SUB * 4)

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// MB rows of x (blockIdx.y names which) against R features a block.  A thread owns a (feature, chunk) pair at a time and walks
// its 128 k's; 128 such pairs go through the ring side by side, 32 k's a stage, copied so that eight lanes take a 128-byte line.
// The ring's first stages are asked for before the kernel before this one has ended: no kernel writes weights.
// Bound: the weights' bytes.  Two blocks an SM keep 96 KB in flight.  A warp's pairs are of neighbouring features, so that its
// lanes read few places of x and not 32, and a whole stage's reads run ahead of its sums.  Before (pairs of neighbouring chunks, a
// question before every four k's, three stages padded to 144 bytes a pair, x by way of registers), in us, before / now:
//   rows    2560 x 2048    2048 x 2048    11264 x 2048    2048 x 5632    32000 x 2048    2048 x 14336
//      1      8.0 / 5.6      5.5 / 5.6     19.1 / 18.6    12.9 / 11.9     51.6 / 45.8     62.5 / 26.6
//      2     10.4 / 6.0      7.2 / 5.7     22.9 / 17.9    16.6 / 12.5     60.8 / 46.6      124 / 46.7
//      8     21.2 / 15.0    14.8 / 13.5    67.9 / 42.9    64.2 / 41.5      151 / 102       452 / 165
template <int MB, int STAGES>
__global__ void __launch_bounds__(GEMV_THREADS)
gemv_f32_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, int ldw, float* __restrict__ out, int ldo,
                int M, int N, int K, int R) {
  extern __shared__ __align__(16) float sm[];
  const int nch = (K + KCHUNK - 1) / KCHUNK;
  float* ring = sm;
  float* xs = ring + STAGES * GEMV_THREADS * GEMV_SUB;  // [MB][nch][GEMV_XCHUNK]
  float* part = xs + MB * nch * GEMV_XCHUNK;                 // [MB][nch * rows]
  const int tid = threadIdx.x;
  const int n0 = blockIdx.x * R, rows = min(R, N - n0);
  const int m0 = blockIdx.y * MB, mb = min(MB, M - m0);
  const int items = rows * nch, most = R * nch;
  const int steps = (items + GEMV_THREADS - 1) / GEMV_THREADS * (KCHUNK / GEMV_SUB);
  pdl_trigger();

  // eight 16-byte pieces a thread and stage: piece tid % 8 of items tid / 8 + 16 j
  const int piece = (tid & 7) * 4, swizzled = ((tid & 7) ^ (tid / 8 & 7)) * 4;
  const float* src[8];
  int k_at[8];
  auto load = [&](int step) {
    const int sub = step % (KCHUNK / GEMV_SUB);
    float* dst = ring + (size_t)(step % STAGES) * GEMV_THREADS * GEMV_SUB;
    if (sub == 0) {
      const int base = step / (KCHUNK / GEMV_SUB) * GEMV_THREADS + tid / 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int item = base + 16 * j;
        const int c = item / rows, r = item - c * rows;
        k_at[j] = item < items ? c * KCHUNK + piece : K;
        src[j] = w + (size_t)(n0 + r) * ldw + c * KCHUNK + piece;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (k_at[j] + sub * GEMV_SUB < K) cp_async16(dst + (tid / 8 + 16 * j) * GEMV_SUB + swizzled, src[j] + sub * GEMV_SUB);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) {
    if (i < steps) load(i);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  pdl_wait();
#pragma unroll
  for (int m = 0; m < MB; ++m)
    for (int k = tid * 4; k < K; k += GEMV_THREADS * 4) {
      float* at = xs + (m * nch + k / KCHUNK) * GEMV_XCHUNK + k % KCHUNK;
      if (m < mb) cp_async16(at, x + (size_t)(m0 + m) * ldx + k);
      else *reinterpret_cast<float4*>(at) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");  // (the ring's first stages too: they were asked for long before)

  float acc[MB];
#pragma unroll
  for (int m = 0; m < MB; ++m) acc[m] = 0.f;
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // everyone's pieces of this stage (and, first, x) are there, and the stage before it is free
    if (step + STAGES - 1 < steps) load(step + STAGES - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const int sub = step % (KCHUNK / GEMV_SUB);
    const int item = step / (KCHUNK / GEMV_SUB) * GEMV_THREADS + tid;
    const int c = min(item, items - 1) / rows;
    const float* wr = ring + (size_t)(step % STAGES) * GEMV_THREADS * GEMV_SUB + tid * GEMV_SUB;
    const float* xr = xs + c * GEMV_XCHUNK + sub * GEMV_SUB;
    const int left = item < items ? (K - c * KCHUNK - sub * GEMV_SUB) : 0;  // k's of this stage that exist (a multiple of 4)
    auto four = [&](int i, const float4& a) {
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        const float4 b = *reinterpret_cast<const float4*>(xr + m * nch * GEMV_XCHUNK + i);
        acc[m] = fmaf(b.x, a.x, acc[m]);
        acc[m] = fmaf(b.y, a.y, acc[m]);
        acc[m] = fmaf(b.z, a.z, acc[m]);
        acc[m] = fmaf(b.w, a.w, acc[m]);
      }
    };
    if (left >= GEMV_SUB) {  // (without a question in between, so that the reads run ahead of the sums)
#pragma unroll
      for (int i = 0; i < GEMV_SUB; i += 4) four(i, *reinterpret_cast<const float4*>(wr + (i ^ (tid & 7) * 4)));
    } else {
      for (int i = 0; i < left; i += 4) four(i, *reinterpret_cast<const float4*>(wr + (i ^ (tid & 7) * 4)));
    }
    if (sub == KCHUNK / GEMV_SUB - 1) {
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        if (item < items) part[m * most + item] = acc[m];
        acc[m] = 0.f;
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < rows * mb; i += GEMV_THREADS) {
    const int m = i / rows, r = i - m * rows;
    float total = 0.f;
#pragma unroll 8
    for (int c = 0; c < nch; ++c) total += part[m * most + c * rows + r];
    out[(size_t)(m0 + m) * ldo + n0 + r] = total;
  }
}

// ------------------------------------------------------------------ 32-bit, many rows
#define GEMM_TK 32
#define GEMM_ROW (GEMM_TK + 4)  // floats per row of a stage: 144 bytes, so that rows next to each other start four banks apart
#define GEMM_STAGES 4
#define GEMM_THREADS 128
static_assert(KCHUNK % GEMM_TK == 0 && KCHUNK % GEMV_SUB == 0, "stages must not straddle the chunks of the summation order");

// A tile of BM x BN outputs by 128 threads, RM x RN of them each: thread (ty, tx) has rows ty + (128 RN / BN) i and columns
// tx + (BN / RN) j, so that a warp's 16-byte reads along k meet all banks.  Three stages of 32 k's are on their way while one is
// multiplied (with one stage ahead in registers, the loads' latency was three quarters of the time).  VEC: rows start on 16
// bytes and K is a multiple of 4; otherwise a stage is put into shared memory number by number.
template <int BM, int BN, int RM, int RN, bool VEC>
__global__ void __launch_bounds__(GEMM_THREADS)
gemm_f32_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, int ldw, float* __restrict__ out, int ldo,
                int M, int N, int K) {
  constexpr int TX = BN / RN, TY = BM / RM, PIECES = GEMM_TK / 4;
  static_assert(TX * TY == GEMM_THREADS && (BM + BN) * PIECES % GEMM_THREADS == 0, "a stage must be whole loads of every thread");
  extern __shared__ __align__(16) float sm[];  // [STAGES][BM + BN][GEMM_ROW]
  const int tid = threadIdx.x, ty = tid / TX, tx = tid % TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  auto load = [&](int t) {
    float* stage = sm + (size_t)(t % GEMM_STAGES) * (BM + BN) * GEMM_ROW;
#pragma unroll
    for (int j = 0; j < (BM + BN) * PIECES / GEMM_THREADS; ++j) {
      const int i = tid + j * GEMM_THREADS, row = i / PIECES, k = t * GEMM_TK + i % PIECES * 4;
      const bool is_x = row < BM;
      const int r = is_x ? m0 + row : n0 + row - BM;
      const bool here = r < (is_x ? M : N);
      const float* src = is_x ? x + (size_t)(here ? r : 0) * ldx + k : w + (size_t)(here ? r : 0) * ldw + k;
      float* dst = stage + row * GEMM_ROW + i % PIECES * 4;
      if (VEC) {  // zeros for what does not exist
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                     "l"(here && k < K ? src : (is_x ? x : w)), "r"(here && k < K ? 16 : 0) : "memory");
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[e] = (here && k + e < K) ? src[e] : 0.f;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[RM][RN], total[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = total[i][j] = 0.f;
  const int tiles = (K + GEMM_TK - 1) / GEMM_TK;
#pragma unroll
  for (int t = 0; t < GEMM_STAGES - 1; ++t) {
    if (t < tiles) load(t);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int t = 0; t < tiles; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GEMM_STAGES - 2) : "memory");
    __syncthreads();  // this stage is there for everyone, and everyone has left the one that is loaded next
    if (t + GEMM_STAGES - 1 < tiles) load(t + GEMM_STAGES - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const float* xs = sm + (size_t)(t % GEMM_STAGES) * (BM + BN) * GEMM_ROW;
    const float* ws = xs + BM * GEMM_ROW;
#pragma unroll
    for (int k = 0; k < GEMM_TK; k += 4) {
      float4 a[RM], b[RN];
#pragma unroll
      for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + (ty + TY * i) * GEMM_ROW + k);
#pragma unroll
      for (int j = 0; j < RN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + (tx + TX * j) * GEMM_ROW + k);
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    if ((t + 1) % (KCHUNK / GEMM_TK) == 0 || t + 1 == tiles) {
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          total[i][j] += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int m = m0 + ty + TY * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      const int n = n0 + tx + TX * j;
      if (n < N) out[(size_t)m * ldo + n] = total[i][j];
    }
  }
}

template <int MB, int STAGES>
static int launch_gemv_f32(const float* x, int ldx, const float* w, int ldw, float* out, int ldo, int M, int N, int K, int R,
                           size_t smem, cudaStream_t stream) {
  auto kern = gemv_f32_kernel<MB, STAGES>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    RL_REFUSE(4, "gemm_f32: cannot get %zu bytes of shared memory", smem);
  dim3 grid((N + R - 1) / R, (M + MB - 1) / MB);
  RL_LAUNCH_CHECK(rl_launch(kern, grid, GEMV_THREADS, smem, stream, x, ldx, w, ldw, out, ldo, M, N, K, R));
  return 0;
}

template <int BM, int BN, int RM, int RN>
static int launch_gemm_f32(const float* x, int ldx, const float* w, int ldw, float* out, int ldo, int M, int N, int K, bool vec,
                           cudaStream_t stream) {
  const int gy = (M + BM - 1) / BM;
  if (gy > 65535) RL_REFUSE(3, "gemm_f32: %d rows exceed %d", M, 65535 * BM);
  constexpr int smem = GEMM_STAGES * (BM + BN) * GEMM_ROW * 4;
  dim3 grid((N + BN - 1) / BN, gy);
  auto kern = vec ? gemm_f32_kernel<BM, BN, RM, RN, true> : gemm_f32_kernel<BM, BN, RM, RN, false>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    RL_REFUSE(5, "gemm_f32: cannot get %d bytes of shared memory", smem);
  kern<<<grid, GEMM_THREADS, smem, stream>>>(x, ldx, w, ldw, out, ldo, M, N, K);
  RL_LAUNCH_RESULT();
}

static size_t gemv_f32_smem(int stages, int mb, int nch, int R) {
  return (size_t)stages * GEMV_STAGE_BYTES + (size_t)mb * nch * (GEMV_XCHUNK + R) * sizeof(float);
}

// How the few rows of a product are streamed: mb rows of x a block (0: not at all), R features a block, the ring's stages.
struct GemvPlan {
  int mb, R, stages;
  size_t smem;
};
static GemvPlan gemv_f32_plan(int M, int N, int K, int sms) {
  const int nch = (K + KCHUNK - 1) / KCHUNK;
  const size_t half = 112 * 1024, third = 74 * 1024, whole = 224 * 1024;
  // features whose sums a block has room for beside a ring of three stages and its rows of x
  auto room = [&](int mb, size_t limit) {
    const long long sums = ((long long)limit - 3 * GEMV_STAGE_BYTES) / (4LL * mb * nch) - GEMV_XCHUNK;
    return (int)(nch <= GEMV_MAX_ITEMS && sums > GEMV_MAX_ITEMS / nch ? GEMV_MAX_ITEMS / nch : sums);
  };
  // features a block: as many as make one wave of per_sm blocks an SM, or where a block has no room for those, of as few equal waves as it takes
  auto features = [&](int per_sm, int most) {
    const int R = (N + per_sm * sms - 1) / (per_sm * sms), waves = (R + most - 1) / most;
    return (R + waves - 1) / waves;
  };
  auto walk = [&](int per_sm, int R) {  // passes of 128 pairs on the busiest SM
    const long long waves = ((N + R - 1) / R + (long long)per_sm * sms - 1) / (per_sm * sms);
    return waves * per_sm * ((R * nch + GEMV_THREADS - 1) / GEMV_THREADS);
  };
  // As many rows of x a block as there are, up to four, while two blocks of a few features fit an SM: blocks of fewer rows read all weights
  // again (four rows of 128256 x 2048: 212 us with four rows a block, 360 with two; of 16384 x 3712, where a block of four has room for nine
  // features, 72 and 144).  Else one row, and at last one block an SM (up to 338 chunks: K of 43264).
  const int wave = (N + 2 * sms - 1) / (2 * sms), few = wave < GEMV_FEW ? wave : GEMV_FEW;
  int mb = M == 1 ? 1 : M == 2 ? 2 : 4;
  while (mb > 1 && room(mb, half) < few) mb /= 2;
  const bool two = room(mb, half) >= few;
  const size_t limit = two ? half : whole;
  const int most = room(mb, limit), most3 = two ? room(mb, third) : 0;
  if (most < 1) return {0, 0, 0, 0};
  int R = features(two ? 2 : 1, most), stages = gemv_f32_smem(4, mb, nch, R) > limit ? 3 : 4;
  // three blocks an SM where that is less to walk through (2560 x 2048 with 2 rows: 9 features of 16 chunks are 144 pairs, two passes of 128; 6
  // are one: 7.9 and 6.0 us)
  if (most3 >= 1 && walk(3, features(3, most3)) < walk(2, R)) R = features(3, most3), stages = 3;
  return {mb, R, stages, gemv_f32_smem(stages, mb, nch, R)};
}
// Rows of x that a block takes beside the weights, or 0 where the product goes by tiles (operands in 16-byte pieces).
RL_API int rl_gemm_f32_streams(int M, int N, int K, int sms) { return M > 0 && M <= GEMV_ROWS && N > 0 && K > 0 && sms > 0 ? gemv_f32_plan(M, N, K, sms).mb : 0; }

RL_API int rl_gemm_f32(const float* x, int ldx, const float* w, int ldw, float* out, int ldo, int M, int N, int K, int sms,
                       cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || sms <= 0) RL_REFUSE(1, "gemm_f32: M=%d N=%d K=%d on %d SMs", M, N, K, sms);
  if (ldx < K || ldw < K || ldo < N) RL_REFUSE(2, "gemm_f32: leading sizes %d/%d/%d too small", ldx, ldw, ldo);
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  const GemvPlan p = M <= GEMV_ROWS && vec ? gemv_f32_plan(M, N, K, sms) : GemvPlan{};
  if (p.mb > 0) {
#define RL_GEMV(MB, STAGES) return launch_gemv_f32<MB, STAGES>(x, ldx, w, ldw, out, ldo, M, N, K, p.R, p.smem, stream)
    if (p.mb == 1 && p.stages == 4) RL_GEMV(1, 4);
    if (p.mb == 1) RL_GEMV(1, 3);
    if (p.mb == 2 && p.stages == 4) RL_GEMV(2, 4);
    if (p.mb == 2) RL_GEMV(2, 3);
    if (p.stages == 4) RL_GEMV(4, 4);
    RL_GEMV(4, 3);
#undef RL_GEMV
  }
  // the tile with the least work on the busiest SM: its blocks there, times the tile's outputs, times what an output costs with
  // that many outputs a thread (shared-memory reads per FMA)
  const int tile[4][2] = {{64, 64}, {64, 32}, {32, 32}, {128, 64}};
  const float cost[4] = {1.05f, 1.2f, 1.5f, 1.0f};
  int best = 0;
  float least = INFINITY;
  for (int i = 0; i < 4; ++i) {
    const long long blocks = (long long)((M + tile[i][0] - 1) / tile[i][0]) * ((N + tile[i][1] - 1) / tile[i][1]);
    const float c = (float)((blocks + sms - 1) / sms) * tile[i][0] * tile[i][1] * cost[i];
    if (c < least) least = c, best = i;
  }
  if (best == 0) return launch_gemm_f32<64, 64, 8, 4>(x, ldx, w, ldw, out, ldo, M, N, K, vec, stream);
  if (best == 1) return launch_gemm_f32<64, 32, 4, 4>(x, ldx, w, ldw, out, ldo, M, N, K, vec, stream);
  if (best == 2) return launch_gemm_f32<32, 32, 4, 2>(x, ldx, w, ldw, out, ldo, M, N, K, vec, stream);
  return launch_gemm_f32<128, 64, 8, 8>(x, ldx, w, ldw, out, ldo, M, N, K, vec, stream);
}

// bfloat16 operands of any k and any alignment; out_dtype bfloat16 or float32.
RL_API int rl_gemm_bf16_any(const bf16* x, int ldx, const bf16* w, int ldw, void* out, int out_dtype, int ldo, int M,
                            int N, int K, int swiglu, float act_alpha, float act_limit, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) RL_REFUSE(1, "gemm_bf16_any: M=%d N=%d K=%d", M, N, K);
  if (swiglu && (N & 1)) RL_REFUSE(4, "gemm_bf16_any: %d rows of gate and up are not pairs", N);
  if (ldx < K || ldw < K || ldo < (swiglu ? N / 2 : N)) RL_REFUSE(2, "gemm_bf16_any: leading sizes %d/%d/%d too small", ldx, ldw, ldo);
  const int gy = (M + TM - 1) / TM;
  if (gy > 65535) RL_REFUSE(3, "gemm_bf16_any: %d rows exceed %d", M, 65535 * TM);
  dim3 grid((N + TN - 1) / TN, gy);
#define RL_ANY(TO, SW) gemm_fma_kernel<bf16, TO, SW><<<grid, 256, 0, stream>>>(x, ldx, w, ldw, (TO*)out, ldo, M, N, K, act_alpha, act_limit)
  if (out_dtype == RL_BF16 && swiglu) RL_ANY(bf16, true);
  else if (out_dtype == RL_BF16) RL_ANY(bf16, false);
  else if (out_dtype == RL_F32 && swiglu) RL_ANY(float, true);
  else if (out_dtype == RL_F32) RL_ANY(float, false);
  else RL_REFUSE(5, "gemm_bf16_any: unknown output dtype %d", out_dtype);
#undef RL_ANY
  RL_LAUNCH_RESULT();
}
