// Linear attention whose decay and input strength change from token to token, through a 32-bit state per sequence:
//
//   S_t = diag(a_t) S_(t-1) + b_t k_t v_t^T,   o_t = S_t^T (c q_t)        per head; S is [dim, vcols]
//
// a_t = exp(log_decay_t) is one number per key channel (a row of `dim`) or one per head; b_t is one number per head or 1;
// c is a constant.  q and k may have fewer heads than v (`qk_heads`: head h reads q/k head h / (H / qk_heads)).  With `ext` the state has one more column that is fed with v = 1: it carries n_t = a_t n_(t-1) + b_t k_t,
// and the output's last column is n_t . q_t, the normaliser of a matrix memory.  Three kinds of layer use it:
//
//   gated linear attention   a_t = sigmoid(z_t)^(1/tau) per channel (`gla_log_decay` makes log a_t), b = 1
//   state-space layer        a_t = exp(-rate_h dt_t), b_t = dt_t per head, q and k shared by groups of heads (csrc/state_space.cu)
//   matrix memory (mLSTM)    log gates i_t, f_t per head with a running maximum m_t = max(f_t + m_(t-1), i_t):
//                            a_t = exp(f_t + m_(t-1) - m_t), b_t = exp(i_t - m_t) (`mlstm_gates`), `ext` column,
//                            o_t / (max(|n_t . q_t|, exp(-m_t)) + c_den) in `head_norm_gate`
//
// The kernels:
//   gla_log_decay     log a = logsigmoid(z + bias) / tau, 32-bit, from the projection in the run's element type
//   mlstm_gates       the capped log gates, the running maximum through the sequences' records, a's logarithm, b and m per token
//   gated_attn        the recurrence token by token (decode steps, 32-bit runs, short prompts): equal bits however a sequence is cut
//   gated_attn chunked   prompts of bfloat16 runs: chunks of 64 tokens, sub-chunks of 16 (see below; a decay per channel on the tensor
//                     cores, gated_chunk_mma.cuh)
//   head_norm_gate    per head: the normaliser, the RMS norm over the head's values, weight, gate; writes the run's element type
//
// Everything between the projections and the state is 32-bit: decays and their logarithms, gates, the maximum, the state, the sums.
#include "common.cuh"

RL_DEFINE_ERROR_TEXT()

// Every kernel here may start while its predecessors are still running (see pdl_wait), so whatever another kernel or a copy
// writes is read through L2, never through the read-only path.
template <typename T>
__device__ __forceinline__ float gr_load(const T* p) { return to_f32(__ldcg(p)); }

__device__ __forceinline__ float gr_logistic(float x) { return logistic_no_branch(x); }
__device__ __forceinline__ float gr_log_logistic(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// Four neighbouring numbers of a row, `left` of them there (the others are zero); `wide`: the row's start and its length allow one load.
template <typename T>
__device__ __forceinline__ float4 gr_load4(const T* __restrict__ p, int left, bool wide) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (wide && left >= 4) {
    if (sizeof(T) == 4) {
      v = __ldcg(reinterpret_cast<const float4*>(p));
    } else {
      const uint2 u = __ldcg(reinterpret_cast<const uint2*>(p));
      v = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
    }
  } else {
    if (left > 0) v.x = gr_load(p);
    if (left > 1) v.y = gr_load(p + 1);
    if (left > 2) v.z = gr_load(p + 2);
    if (left > 3) v.w = gr_load(p + 3);
  }
  return v;
}
// ---------------------------------------------------------------- log decay of gated linear attention
// Four numbers a thread (of the row's last thread, what is left).  Number by number, with a 64-bit division for each one's row, it
// took 20 us for 2048 rows of 2048; now 11, of which memory's work is 4.
template <typename T>
__global__ void gla_log_decay_kernel(const T* __restrict__ z, int z_stride, const float* __restrict__ bias, float inv_tau,
                                     float* __restrict__ out, int n, long long quads, int wide) {
  pdl_trigger();
  pdl_wait();
  const int n4 = (n + 3) / 4;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < quads; idx += (long long)gridDim.x * blockDim.x) {
    const long long t = quads <= 0x7fffffffLL ? (long long)((unsigned)idx / (unsigned)n4) : idx / n4;
    const int i = (int)(idx - t * n4) * 4, left = n - i;
    float4 v = gr_load4(z + t * z_stride + i, left, wide);
    if (bias) {
      v.x += bias[i];
      if (left > 1) v.y += bias[i + 1];
      if (left > 2) v.z += bias[i + 2];
      if (left > 3) v.w += bias[i + 3];
    }
    v = make_float4(gr_log_logistic(v.x) * inv_tau, gr_log_logistic(v.y) * inv_tau, gr_log_logistic(v.z) * inv_tau, gr_log_logistic(v.w) * inv_tau);
    float* to = out + t * n + i;
    if (wide && left >= 4) {
      *reinterpret_cast<float4*>(to) = v;
    } else {
      to[0] = v.x;
      if (left > 1) to[1] = v.y;
      if (left > 2) to[2] = v.z;
      if (left > 3) to[3] = v.w;
    }
  }
}

RL_API int rl_gla_log_decay(const void* z, int dtype, int z_stride, const float* bias, float tau, float* out, int n_tokens, int n,
                            cudaStream_t stream) {
  if (n_tokens <= 0 || n <= 0 || !(tau > 0.f)) RL_REFUSE(1, "gla_log_decay: T=%d n=%d tau=%g", n_tokens, n, (double)tau);
  const long long quads = (long long)n_tokens * ((n + 3LL) / 4);
  long long blocks = (quads + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  const int wide = n % 4 == 0 && z_stride % 4 == 0 && ((uintptr_t)z & (dtype == RL_BF16 ? 7 : 15)) == 0 && ((uintptr_t)out & 15) == 0;
  if (dtype == RL_BF16)
    RL_LAUNCH_CHECK(rl_launch(gla_log_decay_kernel<bf16>, (int)blocks, 256, 0, stream, (const bf16*)z, z_stride, bias, 1.0f / tau, out, n, quads, wide));
  else if (dtype == RL_F32)
    RL_LAUNCH_CHECK(rl_launch(gla_log_decay_kernel<float>, (int)blocks, 256, 0, stream, (const float*)z, z_stride, bias, 1.0f / tau, out, n, quads, wide));
  else
    RL_REFUSE(2, "gla_log_decay: unknown dtype %d", dtype);
  return 0;
}

// ---------------------------------------------------------------- the gates of a matrix memory
// One warp per (sequence, head).  32 tokens' gates are computed side by side; the running maximum then goes through them in
// order (one lane's values at a time, by shuffle), so its bits do not depend on where a step starts.
template <typename T>
__global__ void mlstm_gates_kernel(const T* __restrict__ gi, const T* __restrict__ gf, int in_stride, const float* __restrict__ bias_i,
                                   const float* __restrict__ bias_f, float cap, float* __restrict__ m_state, const int* __restrict__ slot_ids,
                                   const int* __restrict__ seq_start, float* __restrict__ log_a, float* __restrict__ b_out,
                                   float* __restrict__ m_out, int H) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x;
  const int s = blockIdx.x / H, h = blockIdx.x % H;
  const int t0 = __ldcg(seq_start + s), t1 = __ldcg(seq_start + s + 1);
  float* mp = m_state + (size_t)__ldcg(slot_ids + s) * H + h;
  float m = __ldcg(mp);
  const float bi = bias_i ? bias_i[h] : 0.f, bf = bias_f ? bias_f[h] : 0.f;
  const float inv_cap = 1.0f / cap;
  for (int base = t0; base < t1; base += 32) {
    const int t = base + lane;
    float li = 0.f, lf = 0.f;
    if (t < t1) {
      li = cap * tanhf((gr_load(gi + (size_t)t * in_stride + h) + bi) * inv_cap);
      lf = gr_log_logistic(cap * tanhf((gr_load(gf + (size_t)t * in_stride + h) + bf) * inv_cap));
    }
    const int n = min(32, t1 - base);
    float la = 0.f, bb = 0.f, mo = 0.f;
    for (int j = 0; j < n; ++j) {
      const float lij = __shfl_sync(0xffffffffu, li, j), lfj = __shfl_sync(0xffffffffu, lf, j);
      const float m_new = fmaxf(lfj + m, lij);
      if (lane == j) {
        la = lfj + m - m_new;
        bb = expf(lij - m_new);
        mo = m_new;
      }
      m = m_new;
    }
    if (t < t1) {
      log_a[(size_t)t * H + h] = la;
      b_out[(size_t)t * H + h] = bb;
      m_out[(size_t)t * H + h] = mo;
    }
  }
  if (lane == 0) *mp = m;
}

// The same for long prompts: a block of MG_WARPS warps per (sequence, head) takes 32 MG_WARPS tokens at a time.  A token is the map
// m -> max(m + f, i); two maps in a row are again such a map, (f1, i1) then (f2, i2) = (f1 + f2, max(i1 + f2, i2)), so a warp
// composes its 32 maps by a scan of five shuffles, the warps' totals go through shared memory, and every token applies its
// composed map to the maximum that entered the round.  The sums of f are taken in another order than token by token: equal
// within rounding, not in bits, and the order depends on where the step starts.
#define MG_WARPS 8

template <typename T>
__global__ void __launch_bounds__(32 * MG_WARPS)
mlstm_gates_scan_kernel(const T* __restrict__ gi, const T* __restrict__ gf, int in_stride, const float* __restrict__ bias_i,
                        const float* __restrict__ bias_f, float cap, float* __restrict__ m_state, const int* __restrict__ slot_ids,
                        const int* __restrict__ seq_start, float* __restrict__ log_a, float* __restrict__ b_out,
                        float* __restrict__ m_out, int H) {
  __shared__ float tot_f[MG_WARPS], tot_i[MG_WARPS];
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s = blockIdx.x / H, h = blockIdx.x % H;
  const int t0 = __ldcg(seq_start + s), t1 = __ldcg(seq_start + s + 1);
  float* mp = m_state + (size_t)__ldcg(slot_ids + s) * H + h;
  float m_in = __ldcg(mp);
  const float bi = bias_i ? bias_i[h] : 0.f, bf = bias_f ? bias_f[h] : 0.f;
  const float inv_cap = 1.0f / cap;
  for (int base = t0; base < t1; base += 32 * MG_WARPS) {
    const int t = base + threadIdx.x;
    float li = -INFINITY, lf = 0.f;  // past the end: the map that changes nothing
    if (t < t1) {
      li = cap * tanhf((gr_load(gi + (size_t)t * in_stride + h) + bi) * inv_cap);
      lf = gr_log_logistic(cap * tanhf((gr_load(gf + (size_t)t * in_stride + h) + bf) * inv_cap));
    }
    float F = lf, I = li;  // the tokens of this warp up to and with this lane's, as one map
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float Fp = __shfl_up_sync(0xffffffffu, F, o), Ip = __shfl_up_sync(0xffffffffu, I, o);
      if (lane >= o) {
        I = fmaxf(Ip + F, I);
        F = Fp + F;
      }
    }
    if (lane == 31) {
      tot_f[warp] = F;
      tot_i[warp] = I;
    }
    __syncthreads();
    float m_w = m_in;  // the maximum that enters this warp's tokens
    for (int w = 0; w < warp; ++w) m_w = fmaxf(m_w + tot_f[w], tot_i[w]);
    const float m_new = fmaxf(m_w + F, I);
    float m_prev = __shfl_up_sync(0xffffffffu, m_new, 1);
    if (lane == 0) m_prev = m_w;
    if (t < t1) {
      log_a[(size_t)t * H + h] = lf + m_prev - m_new;
      b_out[(size_t)t * H + h] = expf(li - m_new);
      m_out[(size_t)t * H + h] = m_new;
    }
    for (int w = warp; w < MG_WARPS; ++w) m_w = fmaxf(m_w + tot_f[w], tot_i[w]);  // the maximum after the round, in every thread
    m_in = m_w;
    __syncthreads();
  }
  if (threadIdx.x == 0) *mp = m_in;
}

RL_API int rl_mlstm_gates(const void* gi, const void* gf, int dtype, int in_stride, const float* bias_i, const float* bias_f, float cap,
                          float* m_state, const int* slot_ids, const int* seq_start, float* log_a, float* b_out, float* m_out,
                          int n_seqs, int H, int scan, cudaStream_t stream) {
  if (n_seqs <= 0 || H <= 0 || !(cap > 0.f)) RL_REFUSE(1, "mlstm_gates: S=%d H=%d cap=%g", n_seqs, H, (double)cap);
  if (scan) {
    if (dtype == RL_BF16)
      RL_LAUNCH_CHECK(rl_launch(mlstm_gates_scan_kernel<bf16>, n_seqs * H, 32 * MG_WARPS, 0, stream, (const bf16*)gi, (const bf16*)gf, in_stride,
                                bias_i, bias_f, cap, m_state, slot_ids, seq_start, log_a, b_out, m_out, H));
    else if (dtype == RL_F32)
      RL_LAUNCH_CHECK(rl_launch(mlstm_gates_scan_kernel<float>, n_seqs * H, 32 * MG_WARPS, 0, stream, (const float*)gi, (const float*)gf,
                                in_stride, bias_i, bias_f, cap, m_state, slot_ids, seq_start, log_a, b_out, m_out, H));
    else
      RL_REFUSE(2, "mlstm_gates: unknown dtype %d", dtype);
    return 0;
  }
  if (dtype == RL_BF16)
    RL_LAUNCH_CHECK(rl_launch(mlstm_gates_kernel<bf16>, n_seqs * H, 32, 0, stream, (const bf16*)gi, (const bf16*)gf, in_stride, bias_i, bias_f,
                              cap, m_state, slot_ids, seq_start, log_a, b_out, m_out, H));
  else if (dtype == RL_F32)
    RL_LAUNCH_CHECK(rl_launch(mlstm_gates_kernel<float>, n_seqs * H, 32, 0, stream, (const float*)gi, (const float*)gf, in_stride, bias_i,
                              bias_f, cap, m_state, slot_ids, seq_start, log_a, b_out, m_out, H));
  else
    RL_REFUSE(2, "mlstm_gates: unknown dtype %d", dtype);
  return 0;
}

// ---------------------------------------------------------------- the recurrence, token by token
// A block owns 32 columns of one head's state for one sequence: lane = column, warp w holds rows 32 w .. 32 w + 31 of those
// columns in registers.  Tokens are taken GR_TOK at a time: their q, b k and a (whole head) and v (the block's columns) go to
// shared memory, every warp runs the tokens through its rows, and the warps' partial results are added in warp order.  The
// order of every sum is fixed by the sizes alone.
#define GR_TOK 16

template <typename T>
__global__ void gated_attn_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, int in_stride,
                                  const float* __restrict__ log_decay, int per_channel, const float* __restrict__ in_scale, float q_scale,
                                  float* __restrict__ state, const int* __restrict__ slot_ids, const int* __restrict__ seq_start,
                                  float* __restrict__ out, int out_stride, int H, int QH, int dim, int vdim, int ext) {
  extern __shared__ float sm[];
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int s = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * 32, qh = h / (H / QH);
  const int vcols = vdim + ext;
  const int col = col0 + lane;
  const bool col_ok = col < vcols;
  float* q_s = sm;                      // [GR_TOK][dim]
  float* k_s = q_s + GR_TOK * dim;      // [GR_TOK][dim], times b
  float* a_s = k_s + GR_TOK * dim;      // [GR_TOK][dim]
  float* v_s = a_s + GR_TOK * dim;      // [GR_TOK][32]
  float* part = v_s + GR_TOK * 32;      // [nw][GR_TOK][32]
  const int t0 = __ldcg(seq_start + s), t1 = __ldcg(seq_start + s + 1);
  float* st = state + (((size_t)__ldcg(slot_ids + s) * H + h) * dim) * vcols;
  float S[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const int row = w * 32 + r;
    S[r] = (row < dim && col_ok) ? __ldcg(st + (size_t)row * vcols + col) : 0.f;
  }
  for (int base = t0; base < t1; base += GR_TOK) {
    const int n = min(GR_TOK, t1 - base);
    for (int idx = threadIdx.x; idx < n * dim; idx += blockDim.x) {
      const int j = idx / dim, i = idx - j * dim;
      const int t = base + j;
      const size_t at = (size_t)t * in_stride + (size_t)qh * dim + i;
      const float b = in_scale ? __ldcg(in_scale + (size_t)t * H + h) : 1.f;
      q_s[idx] = gr_load(q + at) * q_scale;
      k_s[idx] = gr_load(k + at) * b;
      a_s[idx] = expf(per_channel ? __ldcg(log_decay + ((size_t)t * H + h) * dim + i) : __ldcg(log_decay + (size_t)t * H + h));
    }
    for (int idx = threadIdx.x; idx < n * 32; idx += blockDim.x) {
      const int j = idx >> 5, c = col0 + (idx & 31);
      float vv = 0.f;
      if (c < vdim) vv = gr_load(v + (size_t)(base + j) * in_stride + (size_t)h * vdim + c);
      else if (c < vcols) vv = 1.f;
      v_s[idx] = vv;
    }
    __syncthreads();
    for (int j = 0; j < n; ++j) {
      const float vj = v_s[j * 32 + lane];
      const float* kj = k_s + j * dim + w * 32;
      const float* qj = q_s + j * dim + w * 32;
      const float* aj = a_s + j * dim + w * 32;
      float o = 0.f;
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        if (w * 32 + r < dim) {
          S[r] = aj[r] * S[r] + kj[r] * vj;
          o += S[r] * qj[r];
        }
      }
      part[(w * GR_TOK + j) * 32 + lane] = o;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < n * 32; idx += blockDim.x) {
      const int j = idx >> 5, c = idx & 31;
      if (col0 + c < vcols) {
        float o = 0.f;
        for (int ww = 0; ww < nw; ++ww) o += part[(ww * GR_TOK + j) * 32 + c];
        out[(size_t)(base + j) * out_stride + (size_t)h * vcols + col0 + c] = o;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const int row = w * 32 + r;
    if (row < dim && col_ok) st[(size_t)row * vcols + col] = S[r];
  }
}

RL_API int rl_gated_attn(const void* q, const void* k, const void* v, int dtype, int in_stride, const float* log_decay, int per_channel,
                         const float* in_scale, float q_scale, float* state, const int* slot_ids, const int* seq_start, float* out,
                         int out_stride, int n_seqs, int H, int QH, int dim, int vdim, int ext, cudaStream_t stream) {
  if (QH <= 0 || H % QH) RL_REFUSE(6, "gated_attn: %d heads are not a multiple of %d q/k heads", H, QH);
  if (n_seqs <= 0 || H <= 0 || dim <= 0 || vdim <= 0 || (ext != 0 && ext != 1) || !log_decay)
    RL_REFUSE(1, "gated_attn: S=%d H=%d dim=%d vdim=%d ext=%d", n_seqs, H, dim, vdim, ext);
  if (dim > 1024) RL_REFUSE(2, "gated_attn: key size %d exceeds 1024", dim);
  const int tiles = (vdim + ext + 31) / 32;
  if (H > 65535 || tiles > 65535) RL_REFUSE(3, "gated_attn: %d heads or %d columns exceed the grid", H, vdim);
  const int nw = (dim + 31) / 32;
  const size_t smem = ((size_t)3 * GR_TOK * dim + GR_TOK * 32 + (size_t)nw * GR_TOK * 32) * sizeof(float);
  if (smem > 227 * 1024) RL_REFUSE(4, "gated_attn: %zu bytes of shared memory", smem);
  dim3 grid(n_seqs, H, tiles);
#define RL_GA(T)                                                                                                                   \
  do {                                                                                                                             \
    if (smem > 48 * 1024) {                                                                                                        \
      cudaError_t e = cudaFuncSetAttribute(gated_attn_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);           \
      if (e != cudaSuccess) RL_REFUSE(4, "gated_attn: %zu bytes of shared memory refused", smem);                                  \
    }                                                                                                                              \
    RL_LAUNCH_CHECK(rl_launch(gated_attn_kernel<T>, grid, nw * 32, smem, stream, (const T*)q, (const T*)k, (const T*)v, in_stride,  \
                              log_decay, per_channel, in_scale, q_scale, state, slot_ids, seq_start, out, out_stride, H, QH, dim,   \
                              vdim, ext));                                                                                               \
  } while (0)
  if (dtype == RL_BF16) RL_GA(bf16);
  else if (dtype == RL_F32) RL_GA(float);
  else RL_REFUSE(5, "gated_attn: unknown dtype %d", dtype);
#undef RL_GA
  return 0;
}

// ---------------------------------------------------------------- the same recurrence, chunk by chunk
// For prompts.  A sequence's tokens are cut into chunks of GC; with n tokens in a chunk, S the state before it,
// A_i = sum_{l <= i} log a_l (per key channel, inside the chunk) and k'_j = b_j k_j:
//   U      = sum_j diag(exp(A_(n-1) - A_j)) k'_j v_j^T                                  (1) what the chunk adds, every chunk at once
//   S_next = diag(exp(A_(n-1))) S + U                                                    (2) the states before every chunk, chunk after chunk
//   o_i    = S^T (q_i * exp(A_i)) + sum_{j<=i} (sum_r q_i[r] k'_j[r] exp(A_i[r] - A_j[r])) v_j   (3) the outputs, every chunk at once
// Only exponents <= 0 occur, whatever the decays are: the scores of (3) between tokens of the same sub-chunk of 16 take
// exp(A_i - A_j) channel by channel; between sub-chunks I > J they factor through the sub-chunks' borders,
//   exp(A_i - A_(16 I - 1)) * exp(A_(16 I - 1) - A_(16 J + 15)) * exp(A_(16 J + 15) - A_j),
// a factor of the query, one of the border pair and one of the key.  All of it is 32-bit FMA arithmetic over a scratch of one
// [dim, vcols] matrix and one row of dim decays per (sequence, head, chunk).  The order of the sums differs from the
// token-by-token kernel's and depends on where the chunks fall, so 32-bit runs keep to the other kernel.
#define GC 64       // tokens per chunk
#define GC_SUB 16   // tokens per sub-chunk
#define GC_COLS 64  // state columns per block
#define GR_LOG2E 1.4426950408889634f

__device__ __forceinline__ float gr_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A last column tile of at most four columns (a matrix memory's normaliser beside values that fill whole tiles) gets no block and
// no round of its own: the block of the tile before it adds those columns up with a thread per (row, quarter of the sum).
__host__ __device__ __forceinline__ int gc_narrow(int vcols) {
  const int tiles = (vcols + GC_COLS - 1) / GC_COLS, rem = vcols - (tiles - 1) * GC_COLS;
  return tiles > 1 && rem <= 4 ? rem : 0;
}

// Rows in shared memory: the key size rounded up to the next odd multiple of four floats, so that rows start on 16 bytes and eight
// neighbouring rows' quarters lie in different banks.  What is past the key size is zero.
__host__ __device__ __forceinline__ int gc_row(int dim) { return ((dim + 3) / 4 | 1) * 4; }

__device__ __forceinline__ float4 gr_times(float4 v, float x) { return make_float4(v.x * x, v.y * x, v.z * x, v.w * x); }
__device__ __forceinline__ void gr_add(float4& acc, float x, const float4& v) {
  acc.x = fmaf(x, v.x, acc.x);
  acc.y = fmaf(x, v.y, acc.y);
  acc.z = fmaf(x, v.z, acc.z);
  acc.w = fmaf(x, v.w, acc.w);
}
__device__ __forceinline__ float gr_dot(const float4& a, const float4& b, float acc) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc)))); }

// Four values of column cc of a tile: the values, then the normaliser's 1, then zeros.
template <typename T>
__device__ __forceinline__ float4 gr_values4(const T* __restrict__ row, int cc, int vdim, int vcols, bool wide) {
  if (cc + 4 <= vdim) return gr_load4(row + cc, 4, wide);
  float4 v = gr_load4(row + cc, vdim - cc, false);
  if (vcols > vdim) {
    const int e = vdim - cc;
    if (e == 0) v.x = 1.f;
    if (e == 1) v.y = 1.f;
    if (e == 2) v.z = 1.f;
    if (e == 3) v.w = 1.f;
  }
  return v;
}
// The values' tile [GC][GC_COLS]; rows from n on are zeros.  All of a thread's loads are asked for before the first is stored.
template <typename T>
__device__ __forceinline__ void gr_load_values(float* v_s, const T* __restrict__ v, size_t in_stride, int col0, int n, int vdim, int vcols, bool wide) {
  constexpr int PER = GC * GC_COLS / 4 / 256;
  float4 x[PER];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int idx = threadIdx.x + 256 * p, i = idx / (GC_COLS / 4), cc = col0 + idx % (GC_COLS / 4) * 4;
    x[p] = i < n ? gr_values4(v + i * in_stride, cc, vdim, vcols, wide) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int p = 0; p < PER; ++p) reinterpret_cast<float4*>(v_s)[threadIdx.x + 256 * p] = x[p];
}

// Bits of `wide` of the two kernels: which rows may be read four numbers at a time.
#define GC_WIDE_QK 1     // q's and k's
#define GC_WIDE_V 2      // v's
#define GC_WIDE_DECAY 4  // the log decays' (per channel)
#define GC_WIDE_STATE 8  // the state's

// (1): grid (S * H, chunks, column tiles), 256 threads: thread (ty, tx) owns rows 4 ty + e and 64 + 4 ty + e of 128 and columns
// 4 tx .. 4 tx + 3, three 16-byte reads of shared memory for 32 multiply-adds.  (Rows ty + 16 a cost nine reads for them, and every
// element of the tiles was loaded by itself, with a division for its row: 76 us for 2048 tokens and 16 heads of 128 x 128, now 53.)
template <typename T>
__global__ void __launch_bounds__(256)
gated_chunk_state_kernel(const T* __restrict__ k, const T* __restrict__ v, int in_stride, const float* __restrict__ log_decay,
                         int per_channel, const float* __restrict__ in_scale, const int* __restrict__ seq_start,
                         float* __restrict__ scratch, float* __restrict__ chunk_decay, int max_chunks, int H, int QH, int dim, int vdim, int ext,
                         int wide) {
  extern __shared__ __align__(16) float sm[];
  pdl_trigger();
  pdl_wait();
  const int s = blockIdx.x / H, h = blockIdx.x % H, c = blockIdx.y, col0 = blockIdx.z * GC_COLS, qh = h / (H / QH);
  const int vcols = vdim + ext;
  const int t0 = __ldcg(seq_start + s) + c * GC;
  const int n = min(GC, __ldcg(seq_start + s + 1) - t0);
  if (n <= 0) return;
  const int DS = gc_row(dim), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* k_s = sm;            // [GC][DS]: first the decays' logarithms, then the weighted keys
  float* v_s = sm + GC * DS;  // [GC][GC_COLS]
  float* v_x = v_s + GC * GC_COLS;  // [GC][4]: the narrow last tile's values
  const int narrow = blockIdx.z == gridDim.z - 1 ? gc_narrow(vcols) : 0;
  const int col_x0 = (int)gridDim.z * GC_COLS;
  const T* vh = v + (size_t)t0 * in_stride + (size_t)h * vdim;
  for (int r = 4 * lane; r < DS; r += 128) {  // a warp a row, eight rows of it at once
    float4 la[GC / 8];
#pragma unroll
    for (int p = 0; p < GC / 8; ++p) {
      const int i = warp + 8 * p;
      const size_t th = (size_t)(t0 + i) * H + h;
      la[p] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < n) {
        if (per_channel) la[p] = gr_load4(log_decay + th * dim + r, dim - r, wide & GC_WIDE_DECAY);
        else la[p].x = la[p].y = la[p].z = la[p].w = __ldcg(log_decay + th);
      }
    }
#pragma unroll
    for (int p = 0; p < GC / 8; ++p) *reinterpret_cast<float4*>(k_s + (warp + 8 * p) * DS + r) = gr_times(la[p], GR_LOG2E);
  }
  for (int idx = threadIdx.x; idx < n * narrow; idx += 256) {
    const int i = idx / narrow, e = idx - i * narrow, cc = col_x0 + e;
    v_x[i * 4 + e] = cc < vdim ? gr_load(vh + (size_t)i * in_stride + cc) : 1.f;
  }
  gr_load_values(v_s, vh, in_stride, col0, n, vdim, vcols, wide & GC_WIDE_V);
  __syncthreads();
  // per channel: what the tokens after token i still take away, and the whole chunk's decay
  for (int r = threadIdx.x; r < dim; r += 256) {
    float after = 0.f;
    for (int i0 = GC - 16; i0 >= 0; i0 -= 16) {
      float la[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) la[e] = k_s[(i0 + e) * DS + r];
#pragma unroll
      for (int e = 15; e >= 0; --e) {
        k_s[(i0 + e) * DS + r] = after;
        after += la[e];
      }
    }
    if (blockIdx.z == 0) chunk_decay[((size_t)blockIdx.x * max_chunks + c) * dim + r] = gr_exp2(after);
  }
  __syncthreads();
  for (int r = 4 * lane; r < DS; r += 128) {
    float4 kv[GC / 8];
#pragma unroll
    for (int p = 0; p < GC / 8; ++p) {
      const int i = warp + 8 * p;
      kv[p] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < n) {
        const float b = in_scale ? __ldcg(in_scale + (size_t)(t0 + i) * H + h) : 1.f;
        kv[p] = gr_times(gr_load4(k + (size_t)(t0 + i) * in_stride + (size_t)qh * dim + r, dim - r, wide & GC_WIDE_QK), b);
      }
    }
#pragma unroll
    for (int p = 0; p < GC / 8; ++p) {
      float4* at = reinterpret_cast<float4*>(k_s + (warp + 8 * p) * DS + r);
      const float4 after = *at;
      *at = make_float4(kv[p].x * gr_exp2(after.x), kv[p].y * gr_exp2(after.y), kv[p].z * gr_exp2(after.z), kv[p].w * gr_exp2(after.w));
    }
  }
  __syncthreads();
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  float* u = scratch + ((size_t)blockIdx.x * max_chunks + c) * dim * vcols;
  for (int r0 = 0; r0 < dim; r0 += 128) {  // 128 rows of the state at a time: eight to a thread
    const int ra = r0 + 4 * ty, rb = ra + 64;
    const bool has_a = ra < dim, has_b = rb < dim;
    float4 acc[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) acc[a] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
      const float4 vv = *reinterpret_cast<const float4*>(v_s + i * GC_COLS + 4 * tx);
      if (has_a) {
        const float4 kv = *reinterpret_cast<const float4*>(k_s + i * DS + ra);
        gr_add(acc[0], kv.x, vv);
        gr_add(acc[1], kv.y, vv);
        gr_add(acc[2], kv.z, vv);
        gr_add(acc[3], kv.w, vv);
      }
      if (has_b) {
        const float4 kv = *reinterpret_cast<const float4*>(k_s + i * DS + rb);
        gr_add(acc[4], kv.x, vv);
        gr_add(acc[5], kv.y, vv);
        gr_add(acc[6], kv.z, vv);
        gr_add(acc[7], kv.w, vv);
      }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int r = (a < 4 ? ra : rb - 4) + a, col = col0 + 4 * tx;
      if (r < dim) {
        float* to = u + (size_t)r * vcols + col;
        if ((wide & GC_WIDE_STATE) && col < vcols) {
          *reinterpret_cast<float4*>(to) = acc[a];
        } else {
          if (col < vcols) to[0] = acc[a].x;
          if (col + 1 < vcols) to[1] = acc[a].y;
          if (col + 2 < vcols) to[2] = acc[a].z;
          if (col + 3 < vcols) to[3] = acc[a].w;
        }
      }
    }
  }
  for (int idx = threadIdx.x; idx < dim * narrow; idx += 256) {
    const int r = idx / narrow, e = idx - r * narrow;
    float acc = 0.f;
    for (int i = 0; i < n; ++i) acc += k_s[i * DS + r] * v_x[i * 4 + e];
    u[(size_t)r * vcols + col_x0 + e] = acc;
  }
}

// (2): one thread per V neighbouring elements of a (sequence, head)'s state; leaves in every chunk's place the state BEFORE that
// chunk.  Memory's work alone (10 us with four elements a thread, 48 with one, for the same case): four wherever rows are whole quarters.
template <int V>
__global__ void gated_chunk_scan_kernel(float* __restrict__ state, const int* __restrict__ slot_ids, const int* __restrict__ seq_start,
                                        float* __restrict__ scratch, const float* __restrict__ chunk_decay, int max_chunks, int H,
                                        int dim, int vcols) {
  struct __align__(4 * V) Some { float x[V]; };
  pdl_trigger();
  pdl_wait();
  const int s = blockIdx.x / H, h = blockIdx.x % H;
  const int elems = dim * vcols;
  const int e = (blockIdx.y * blockDim.x + threadIdx.x) * V;
  if (e >= elems) return;
  const int r = e / vcols;
  const int len = __ldcg(seq_start + s + 1) - __ldcg(seq_start + s);
  float* st = state + ((size_t)__ldcg(slot_ids + s) * H + h) * elems + e;
  float* u = scratch + (size_t)blockIdx.x * max_chunks * elems + e;
  const float* g = chunk_decay + (size_t)blockIdx.x * max_chunks * dim + r;
  auto load = [](const float* p) {
    Some v;
    if constexpr (V == 4) {
      const float4 w = __ldcg(reinterpret_cast<const float4*>(p));
      v.x[0] = w.x; v.x[1] = w.y; v.x[2] = w.z; v.x[3] = w.w;
    } else {
      v.x[0] = __ldcg(p);
    }
    return v;
  };
  Some S = load(st);
  const int n_chunks = (len + GC - 1) / GC;
  for (int c0 = 0; c0 < n_chunks; c0 += 8) {  // eight chunks' additions are asked for at once, then taken in order
    Some add[8];
    float dec[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c0 + j < n_chunks) {
        add[j] = load(u + (size_t)(c0 + j) * elems);
        dec[j] = __ldcg(g + (size_t)(c0 + j) * dim);
      }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c0 + j < n_chunks) {
        *reinterpret_cast<Some*>(u + (size_t)(c0 + j) * elems) = S;
#pragma unroll
        for (int i = 0; i < V; ++i) S.x[i] = dec[j] * S.x[i] + add[j].x[i];
      }
  }
  *reinterpret_cast<Some*>(st) = S;
}

// (3): grid (S * H, chunks), 256 threads.  The scores of the chunk are computed once: those inside the sub-chunks by a thread per two
// pairs of tokens (an exponential per channel) and a quarter of a token with itself, those between sub-chunks by thread (ty, tx) for
// tokens ty + 16 a and tx + 16 b; then, column tile after column tile, outputs for rows ty + 16 a and columns 4 tx .. 4 tx + 3.
// The scores and the values' tile take the place of the decays' sums, and the state's tile the keys' place, once those are used up:
// three tiles of [GC][gc_row(dim)] in all, so that two blocks share an SM at dim = 128.
// Bound: shared memory's reads beside the FMA pipe; so all inner loops take four channels (or tokens) by 16-byte reads: 12 cycles of
// reads for 16 of multiply-adds in the outputs' loops.  With a read per number, half of the threads idle in the sub-chunks' scores and
// the tiles loaded number by number it was 183 us for 2048 tokens and 16 heads of 128 x 128, now 117.
template <typename T>
__global__ void __launch_bounds__(256, 2)
gated_chunk_out_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, int in_stride,
                       const float* __restrict__ log_decay, int per_channel, const float* __restrict__ in_scale, float q_scale,
                       const int* __restrict__ seq_start, const float* __restrict__ scratch, int max_chunks, float* __restrict__ out,
                       int out_stride, int H, int QH, int dim, int vdim, int ext, int wide) {
  extern __shared__ __align__(16) float sm[];
  pdl_trigger();
  pdl_wait();
  const int s = blockIdx.x / H, h = blockIdx.x % H, c = blockIdx.y, qh = h / (H / QH);
  const int vcols = vdim + ext;
  const int t0 = __ldcg(seq_start + s) + c * GC;
  const int n = min(GC, __ldcg(seq_start + s + 1) - t0);
  if (n <= 0) return;
  const int DS = gc_row(dim), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int PS = GC + 4;
  float* q_s = sm;                    // [GC][DS]
  float* k_s = q_s + GC * DS;         // [GC][DS]; later the state's tile [dim][GC_COLS]
  float* a_s = k_s + GC * DS;         // [GC][DS]: A_i in units of log 2; later v_s and p_s
  float* v_s = a_s;                   // [GC][GC_COLS]
  float* p_s = v_s + GC * GC_COLS;    // [GC][PS]
  float* d_s = a_s + max(GC * DS, GC * GC_COLS + GC * PS);  // [5][DS]: the decay over sub-chunk 1 and over sub-chunk 2; A at the ends of sub-chunks 0, 1, 2
  float* v_x = d_s + 5 * DS;          // [GC][4]: the narrow last tile's values
  const int narrow = gc_narrow(vcols), wide_cols = vcols - narrow;
  const T* vh = v + (size_t)t0 * in_stride + (size_t)h * vdim;
  for (int idx = threadIdx.x; idx < n * narrow; idx += 256) {
    const int i = idx / narrow, e = idx - i * narrow, cc = wide_cols + e;
    v_x[i * 4 + e] = cc < vdim ? gr_load(vh + (size_t)i * in_stride + cc) : 1.f;
  }
  for (int r = 4 * lane; r < DS; r += 128) {  // a warp a row, four rows of it at once
    for (int i0 = warp; i0 < GC; i0 += 32) {
      float4 qv[4], kv[4], la[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int i = i0 + 8 * p;
        qv[p] = kv[p] = la[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n) {
          const size_t at = (size_t)(t0 + i) * in_stride + (size_t)qh * dim + r;
          const size_t th = (size_t)(t0 + i) * H + h;
          qv[p] = gr_load4(q + at, dim - r, wide & GC_WIDE_QK);
          kv[p] = gr_load4(k + at, dim - r, wide & GC_WIDE_QK);
          if (per_channel) la[p] = gr_load4(log_decay + th * dim + r, dim - r, wide & GC_WIDE_DECAY);
          else la[p].x = la[p].y = la[p].z = la[p].w = __ldcg(log_decay + th);
          if (in_scale) kv[p] = gr_times(kv[p], __ldcg(in_scale + th));
        }
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int at = (i0 + 8 * p) * DS + r;
        *reinterpret_cast<float4*>(q_s + at) = gr_times(qv[p], q_scale);
        *reinterpret_cast<float4*>(k_s + at) = kv[p];
        *reinterpret_cast<float4*>(a_s + at) = gr_times(la[p], GR_LOG2E);
      }
    }
  }
  __syncthreads();
  for (int r = threadIdx.x; r < DS; r += 256) {  // A_i: the running sum down the chunk (rows past the last token repeat it)
    float run = 0.f;
    for (int i0 = 0; i0 < GC; i0 += 16) {
      float la[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) la[e] = a_s[(i0 + e) * DS + r];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        run += la[e];
        a_s[(i0 + e) * DS + r] = run;
      }
    }
  }
  __syncthreads();
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  // ---- scores inside a sub-chunk: the decay between the two tokens, channel by channel.  The 120 pairs of a sub-chunk's 64 threads
  // are the eight folded rows 15 - f and f of 15 pairs in all.
  float own[2] = {0.f, 0.f}, self = 0.f;
  int own_at[2];
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const int sub = threadIdx.x >> 6, m = (threadIdx.x & 63) + 60 * w, f = m / 15, e = m - 15 * f;
    const bool upper = e < 15 - f;
    const int i = GC_SUB * sub + (upper ? 15 - f : f), j = GC_SUB * sub + (upper ? e : e - (15 - f));
    own_at[w] = (threadIdx.x & 63) < 60 ? i * PS + j : -1;
    if (own_at[w] >= 0) {
      const float *qi = q_s + i * DS, *kj = k_s + j * DS, *ai = a_s + i * DS, *aj = a_s + j * DS;
#pragma unroll 2
      for (int r = 0; r < dim; r += 4) {
        const float4 x = *reinterpret_cast<const float4*>(qi + r), y = *reinterpret_cast<const float4*>(kj + r);
        const float4 a = *reinterpret_cast<const float4*>(ai + r), b = *reinterpret_cast<const float4*>(aj + r);
        own[w] = fmaf(x.x * y.x, gr_exp2(a.x - b.x), own[w]);
        own[w] = fmaf(x.y * y.y, gr_exp2(a.y - b.y), own[w]);
        own[w] = fmaf(x.z * y.z, gr_exp2(a.z - b.z), own[w]);
        own[w] = fmaf(x.w * y.w, gr_exp2(a.w - b.w), own[w]);
      }
    }
  }
  {  // a token with itself: no decay
    const int i = threadIdx.x >> 2;
    for (int r = 4 * (threadIdx.x & 3); r < dim; r += 16)
      self = gr_dot(*reinterpret_cast<const float4*>(q_s + i * DS + r), *reinterpret_cast<const float4*>(k_s + i * DS + r), self);
    self += __shfl_xor_sync(0xffffffffu, self, 1);
    self += __shfl_xor_sync(0xffffffffu, self, 2);
  }
  __syncthreads();
  // ---- queries relative to the start of their sub-chunk, keys relative to the end of theirs, and the two inner sub-chunks' decays
  for (int r = 4 * lane; r < DS; r += 128) {
#pragma unroll 4
    for (int i = warp; i < GC; i += 8) {
      const int sub = i / GC_SUB;
      const float4 mine = *reinterpret_cast<const float4*>(a_s + i * DS + r);
      const float4 end = *reinterpret_cast<const float4*>(a_s + (sub * GC_SUB + GC_SUB - 1) * DS + r);
      float4 before = make_float4(0.f, 0.f, 0.f, 0.f);
      if (sub > 0) before = *reinterpret_cast<const float4*>(a_s + (sub * GC_SUB - 1) * DS + r);
      float4 x = *reinterpret_cast<const float4*>(q_s + i * DS + r), y = *reinterpret_cast<const float4*>(k_s + i * DS + r);
      x.x *= gr_exp2(mine.x - before.x); x.y *= gr_exp2(mine.y - before.y); x.z *= gr_exp2(mine.z - before.z); x.w *= gr_exp2(mine.w - before.w);
      y.x *= gr_exp2(end.x - mine.x); y.y *= gr_exp2(end.y - mine.y); y.z *= gr_exp2(end.z - mine.z); y.w *= gr_exp2(end.w - mine.w);
      *reinterpret_cast<float4*>(q_s + i * DS + r) = x;
      *reinterpret_cast<float4*>(k_s + i * DS + r) = y;
    }
  }
  for (int r = threadIdx.x; r < DS; r += 256) {
    const float a0 = a_s[(GC_SUB - 1) * DS + r], a1 = a_s[(2 * GC_SUB - 1) * DS + r], a2 = a_s[(3 * GC_SUB - 1) * DS + r];
    d_s[r] = gr_exp2(a1 - a0);
    d_s[DS + r] = gr_exp2(a2 - a1);
    d_s[2 * DS + r] = a0;
    d_s[3 * DS + r] = a1;
    d_s[4 * DS + r] = a2;
  }
  __syncthreads();  // the decays' sums are used up from here on
  // ---- scores between sub-chunks
  float p10 = 0.f, p21 = 0.f, p32 = 0.f, p20 = 0.f, p31 = 0.f, p30 = 0.f;
  for (int r = 0; r < dim; r += 4) {
    const float4 q1 = *reinterpret_cast<const float4*>(q_s + (ty + 16) * DS + r), k0 = *reinterpret_cast<const float4*>(k_s + tx * DS + r);
    float4 q2 = *reinterpret_cast<const float4*>(q_s + (ty + 32) * DS + r), q3 = *reinterpret_cast<const float4*>(q_s + (ty + 48) * DS + r);
    const float4 k1 = *reinterpret_cast<const float4*>(k_s + (tx + 16) * DS + r), k2 = *reinterpret_cast<const float4*>(k_s + (tx + 32) * DS + r);
    const float4 d1 = *reinterpret_cast<const float4*>(d_s + r), d2 = *reinterpret_cast<const float4*>(d_s + DS + r);
    p10 = gr_dot(q1, k0, p10);
    p21 = gr_dot(q2, k1, p21);
    p32 = gr_dot(q3, k2, p32);
    q2.x *= d1.x; q2.y *= d1.y; q2.z *= d1.z; q2.w *= d1.w;
    p20 = gr_dot(q2, k0, p20);
    q3.x *= d2.x; q3.y *= d2.y; q3.z *= d2.z; q3.w *= d2.w;
    p31 = gr_dot(q3, k1, p31);
    q3.x *= d1.x; q3.y *= d1.y; q3.z *= d1.z; q3.w *= d1.w;
    p30 = gr_dot(q3, k0, p30);
  }
#pragma unroll
  for (int w = 0; w < 2; ++w)
    if (own_at[w] >= 0) p_s[own_at[w]] = own[w];
  if ((threadIdx.x & 3) == 0) p_s[(threadIdx.x >> 2) * PS + (threadIdx.x >> 2)] = self;
#pragma unroll
  for (int a = 0; a < 4; ++a)
    if (tx > ty) p_s[(ty + 16 * a) * PS + tx + 16 * a] = 0.f;  // (the sub-chunks to the right of a row's own are never read)
  p_s[(ty + 16) * PS + tx] = p10;
  p_s[(ty + 32) * PS + tx] = p20;
  p_s[(ty + 48) * PS + tx] = p30;
  p_s[(ty + 32) * PS + tx + 16] = p21;
  p_s[(ty + 48) * PS + tx + 16] = p31;
  p_s[(ty + 48) * PS + tx + 32] = p32;
  // ---- the queries against the state before the chunk take the whole decay since the chunk's start
  __syncthreads();
  for (int r = 4 * lane; r < DS; r += 128) {
#pragma unroll 2
    for (int i = GC_SUB + warp; i < GC; i += 8) {
      const float4 a = *reinterpret_cast<const float4*>(d_s + (i / GC_SUB + 1) * DS + r);
      float4 x = *reinterpret_cast<const float4*>(q_s + i * DS + r);
      x.x *= gr_exp2(a.x); x.y *= gr_exp2(a.y); x.z *= gr_exp2(a.z); x.w *= gr_exp2(a.w);
      *reinterpret_cast<float4*>(q_s + i * DS + r) = x;
    }
  }
  const float* sp = scratch + ((size_t)blockIdx.x * max_chunks + c) * dim * vcols;
  float* s_s = k_s;  // [dim rounded up to four][GC_COLS]; GC * gc_row(dim) holds it
  const int dim4 = (dim + 3) / 4 * 4;
  for (int col0 = 0; col0 < wide_cols; col0 += GC_COLS) {
    if (col0) __syncthreads();  // the tile before read
    if (wide & GC_WIDE_STATE) {
      for (int idx = threadIdx.x; idx < dim4 * (GC_COLS / 4); idx += 256) {
        const int r = idx / (GC_COLS / 4), cc = col0 + idx % (GC_COLS / 4) * 4;
        const bool here = r < dim && cc < vcols;
        const float* from = here ? sp + (size_t)r * vcols + cc : sp;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(s_s + 4 * idx)), "l"(from), "r"(here ? 16 : 0) : "memory");
      }
    } else {
#pragma unroll 4
      for (int idx = threadIdx.x; idx < dim4 * GC_COLS; idx += 256) {
        const int r = idx / GC_COLS, cc = col0 + idx % GC_COLS;
        s_s[idx] = r < dim && cc < vcols ? __ldcg(sp + (size_t)r * vcols + cc) : 0.f;
      }
    }
    gr_load_values(v_s, vh, in_stride, col0, n, vdim, vcols, wide & GC_WIDE_V);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float4 acc[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[a] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int sub = 0; sub < GC / GC_SUB; ++sub) {
#pragma unroll 1
      for (int j = GC_SUB * sub; j < GC_SUB * (sub + 1); j += 4) {
        float4 vv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) vv[e] = *reinterpret_cast<const float4*>(v_s + (j + e) * GC_COLS + 4 * tx);
#pragma unroll
        for (int a = sub; a < 4; ++a) {
          const float4 pv = *reinterpret_cast<const float4*>(p_s + (ty + 16 * a) * PS + j);
          gr_add(acc[a], pv.x, vv[0]);
          gr_add(acc[a], pv.y, vv[1]);
          gr_add(acc[a], pv.z, vv[2]);
          gr_add(acc[a], pv.w, vv[3]);
        }
      }
    }
#pragma unroll 2
    for (int r = 0; r < dim4; r += 4) {
      float4 t[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) t[e] = *reinterpret_cast<const float4*>(s_s + (r + e) * GC_COLS + 4 * tx);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float4 qv = *reinterpret_cast<const float4*>(q_s + (ty + 16 * a) * DS + r);
        gr_add(acc[a], qv.x, t[0]);
        gr_add(acc[a], qv.y, t[1]);
        gr_add(acc[a], qv.z, t[2]);
        gr_add(acc[a], qv.w, t[3]);
      }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = ty + 16 * a, col = col0 + 4 * tx;
      if (i < n) {
        float* to = out + (size_t)(t0 + i) * out_stride + (size_t)h * vcols + col;
        if ((wide & GC_WIDE_STATE) && col < vcols) {
          *reinterpret_cast<float4*>(to) = acc[a];
        } else {
          if (col < vcols) to[0] = acc[a].x;
          if (col + 1 < vcols) to[1] = acc[a].y;
          if (col + 2 < vcols) to[2] = acc[a].z;
          if (col + 3 < vcols) to[3] = acc[a].w;
        }
      }
    }
  }
  if (narrow > 0) {  // thread (i, part): a quarter of row i's sums over the keys and over the state's rows, added up by shuffles
    const int i = threadIdx.x >> 2, part = threadIdx.x & 3;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int j = part; j <= i; j += 4) {
      const float pv = p_s[i * PS + j];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < narrow) acc[e] += pv * v_x[j * 4 + e];
    }
    for (int r = part; r < dim; r += 4) {
      const float qv = q_s[i * DS + r];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < narrow) acc[e] += qv * __ldcg(sp + (size_t)r * vcols + wide_cols + e);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 1);
      acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 2);
    }
    if (part == 0 && i < n) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < narrow) out[(size_t)(t0 + i) * out_stride + (size_t)h * vcols + wide_cols + e] = acc[e];
    }
  }
}

#include "gated_chunk_mma.cuh"

RL_API long long rl_gated_attn_chunked_scratch_floats(int n_seqs, int max_q_len, int H, int dim, int vcols) {
  return (long long)n_seqs * H * ((max_q_len + GC - 1) / GC) * dim * (vcols + 1);
}

static size_t gated_chunk_out_smem(int dim) {
  const size_t row = gc_row(dim), tile = GC * row, later = (size_t)GC * GC_COLS + GC * (GC + 4);
  return (2 * tile + (tile > later ? tile : later) + 5 * row + GC * 4) * sizeof(float);
}

RL_API int rl_gated_attn_chunked_takes(int dim) { return dim > 0 && gated_chunk_out_smem(dim) <= 227 * 1024; }

// norm_w: null, or the heads' norm weights [vdim]; result is then bfloat16 rows that have been through what head_norm_gate does (gate may
// be null; gate_act as there), where the tensor-core kernels take the call, and nothing is launched and RL_NOT_FUSED returned where
// they do not.  Without it result is float32.
RL_API int rl_gated_attn_chunked(const void* q, const void* k, const void* v, int dtype, int in_stride, const float* log_decay,
                                 int per_channel, const float* in_scale, float q_scale, float* state, const int* slot_ids,
                                 const int* seq_start, float* scratch, void* result, int out_stride, int n_seqs, int max_q_len, int H,
                                 int QH, int dim, int vdim, int ext, const float* norm_w, float eps, const void* gate, int gate_stride,
                                 int gate_act, float out_scale, cudaStream_t stream) {
  if (QH <= 0 || H % QH) RL_REFUSE(6, "gated_attn_chunked: %d heads are not a multiple of %d q/k heads", H, QH);
  if (n_seqs <= 0 || max_q_len <= 0 || H <= 0 || dim <= 0 || vdim <= 0 || (ext != 0 && ext != 1) || !log_decay || !scratch)
    RL_REFUSE(1, "gated_attn_chunked: S=%d max_q=%d H=%d dim=%d vdim=%d ext=%d", n_seqs, max_q_len, H, dim, vdim, ext);
  if (!rl_gated_attn_chunked_takes(dim)) RL_REFUSE(2, "gated_attn_chunked: key size %d needs more shared memory than an SM has", dim);
  const int vcols = vdim + ext;
  const int max_chunks = (max_q_len + GC - 1) / GC, col_tiles = (vcols + GC_COLS - 1) / GC_COLS - (gc_narrow(vcols) > 0 ? 1 : 0);
  const long long sh = (long long)n_seqs * H;
  if (sh > 0x7fffffffLL || max_chunks > 65535 || col_tiles > 65535) RL_REFUSE(3, "gated_attn_chunked: %d chunks or %d column tiles exceed the grid", max_chunks, col_tiles);
  float* chunk_decay = scratch + sh * max_chunks * dim * vcols;
  const int elems = dim * vcols;
  // Rows are read four numbers at a time where each of them starts on four of its type and is whole fours long.
  const uintptr_t four = dtype == RL_BF16 ? 7 : 15;
  float* out = (float*)result;
  int wide = 0;
  if (dim % 4 == 0 && in_stride % 4 == 0 && (((uintptr_t)q | (uintptr_t)k) & four) == 0) wide |= GC_WIDE_QK;
  if (vdim % 4 == 0 && in_stride % 4 == 0 && ((uintptr_t)v & four) == 0) wide |= GC_WIDE_V;
  if (dim % 4 == 0 && ((uintptr_t)log_decay & 15) == 0) wide |= GC_WIDE_DECAY;
  if (vcols % 4 == 0 && (((uintptr_t)state | (uintptr_t)scratch) & 15) == 0 && (norm_w || (out_stride % 4 == 0 && ((uintptr_t)out & 15) == 0))) wide |= GC_WIDE_STATE;
  const int scan_elems = wide & GC_WIDE_STATE ? 4 : 1;
  dim3 grid((unsigned)sh, max_chunks, col_tiles), grid2((unsigned)sh, (elems / scan_elems + 255) / 256), grid3((unsigned)sh, max_chunks);
  if (norm_w && (out_stride % 2 || ((uintptr_t)result & 3) || gate_stride % 2 || ((uintptr_t)gate & 3) || ((uintptr_t)norm_w & 7))) return RL_NOT_FUSED;
  // A decay per channel on bfloat16 rows in 16-byte pieces goes to the tensor cores (gated_chunk_mma.cuh): 2048 tokens, 16 heads of
  // 128 x 128: 98 instead of 185 us for the three steps (117 with the heads' norm and gate, 202 with both behind them).  One decay per head comes with a normaliser column, whose odd rows do not fit.
  if (dtype == RL_BF16 && per_channel && !in_scale && !ext && (wide & GC_WIDE_STATE) && gated_mma_takes(q, k, v, in_stride, log_decay, dim, vdim)) {
#define RL_GM(DP)                                                                                                                     \
  do {                                                                                                                                \
    constexpr size_t s1 = (size_t)GC * (DP + 8) * 4 + GC * (GM_COLS + 8) * 2, s3 = GmOut<DP>::BYTES;                                  \
    if (cudaFuncSetAttribute(gated_mma_state_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1) != cudaSuccess ||      \
        cudaFuncSetAttribute(gated_mma_out_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3) != cudaSuccess)          \
      RL_REFUSE(4, "gated_attn_chunked: %zu bytes of shared memory refused", s3);                                                     \
    RL_LAUNCH_CHECK(rl_launch(gated_mma_state_kernel<DP>, grid3, 256, s1, stream, (const bf16*)k, (const bf16*)v, in_stride, log_decay, \
                              seq_start, scratch, chunk_decay, max_chunks, H, QH, dim, vdim));                                        \
    RL_LAUNCH_CHECK(rl_launch(gated_chunk_scan_kernel<4>, grid2, 256, 0, stream, state, slot_ids, seq_start, scratch,                 \
                              (const float*)chunk_decay, max_chunks, H, dim, vcols));                                                 \
    RL_LAUNCH_CHECK(rl_launch(gated_mma_out_kernel<DP>, grid3, 256, s3, stream, (const bf16*)q, (const bf16*)k, (const bf16*)v,       \
                              in_stride, log_decay, q_scale, seq_start, (const float*)scratch, max_chunks, result, out_stride, H, QH, \
                              dim, vdim, SplNorm{norm_w, eps, (const bf16*)gate, gate_stride, gate_act, out_scale}));                 \
  } while (0)
    if (dim <= 64) RL_GM(64);
    else RL_GM(128);
#undef RL_GM
    return 0;
  }
  if (norm_w) return RL_NOT_FUSED;
  const size_t smem1 = ((size_t)GC * gc_row(dim) + GC * GC_COLS + GC * 4) * sizeof(float), smem3 = gated_chunk_out_smem(dim);
#define RL_GC(T)                                                                                                                     \
  do {                                                                                                                               \
    if (cudaFuncSetAttribute(gated_chunk_state_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1) != cudaSuccess || \
        cudaFuncSetAttribute(gated_chunk_out_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem3) != cudaSuccess)     \
      RL_REFUSE(4, "gated_attn_chunked: %zu bytes of shared memory refused", smem3);                                                 \
    RL_LAUNCH_CHECK(rl_launch(gated_chunk_state_kernel<T>, grid, 256, smem1, stream, (const T*)k, (const T*)v, in_stride, log_decay,  \
                              per_channel, in_scale, seq_start, scratch, chunk_decay, max_chunks, H, QH, dim, vdim, ext, wide));     \
    RL_LAUNCH_CHECK(rl_launch(scan_elems == 4 ? gated_chunk_scan_kernel<4> : gated_chunk_scan_kernel<1>, grid2, 256, 0, stream, state, \
                              slot_ids, seq_start, scratch, (const float*)chunk_decay, max_chunks, H, dim, vcols));                  \
    RL_LAUNCH_CHECK(rl_launch(gated_chunk_out_kernel<T>, grid3, 256, smem3, stream, (const T*)q, (const T*)k, (const T*)v, in_stride,  \
                              log_decay, per_channel, in_scale, q_scale, seq_start, (const float*)scratch, max_chunks, out,          \
                              out_stride, H, QH, dim, vdim, ext, wide));                                                             \
  } while (0)
  if (dtype == RL_BF16) RL_GC(bf16);
  else if (dtype == RL_F32) RL_GC(float);
  else RL_REFUSE(5, "gated_attn_chunked: unknown dtype %d", dtype);
#undef RL_GC
  return 0;
}

// ---------------------------------------------------------------- per head: normaliser, RMS norm, weight, gate
// One warp per (token, head).  x: 32-bit rows of H heads of `xh` numbers, of which the first n are the head's values; with m
// given, x[n] is the head's n . q and the values are first divided by max(|x[n]|, exp(-m)) + den_eps.  Then
//   y_i = v_i / sqrt(mean(v^2) + eps) * weight * act(gate_i)
// weight: [n] shared by the heads, or [H n]; act: 0 none, 1 the logistic function, 2 silu.
// A lane has V neighbouring values at a time: four where all rows start on four and are whole fours long, else one (a matrix memory's
// heads lie an odd number apart).  2048 tokens of 16 heads of 128, with a gate: 17 us with four, 27 with one; memory's work is 5.
#define HN_MAX_PER_LANE 16  // head values up to 512

template <typename T, int V>
__global__ void head_norm_gate_kernel(const float* __restrict__ x, int x_stride, int xh, const float* __restrict__ m, float den_eps,
                                      const float* __restrict__ weight, int weight_per_head, float eps, const T* __restrict__ gate,
                                      int gate_stride, int gate_act, float out_scale, T* __restrict__ out, int out_stride, int n_rows,
                                      int H, int n) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int pair = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (pair >= n_rows * H) return;
  const int t = pair / H, h = pair - t * H;
  const float* xr = x + (size_t)t * x_stride + (size_t)h * xh;
  float inv_den = 1.f;
  if (m != nullptr) inv_den = 1.0f / (fmaxf(fabsf(__ldcg(xr + n)), expf(-__ldcg(m + (size_t)t * H + h))) + den_eps);
  constexpr int GROUPS = HN_MAX_PER_LANE / V;
  const T* g = gate ? gate + (size_t)t * gate_stride + (size_t)h * n : nullptr;
  float vals[GROUPS][V], gates[GROUPS][V];
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < GROUPS; ++e) {
    const int i = V * (lane + 32 * e);
    const bool here = i < n;
    if constexpr (V == 4) {
      const float4 w = here ? gr_load4(xr + i, 4, true) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 y = here && g ? gr_load4(g + i, 4, true) : w;
      vals[e][0] = w.x; vals[e][1] = w.y; vals[e][2] = w.z; vals[e][3] = w.w;
      gates[e][0] = y.x; gates[e][1] = y.y; gates[e][2] = y.z; gates[e][3] = y.w;
    } else {
      vals[e][0] = here ? __ldcg(xr + i) : 0.f;
      gates[e][0] = here && g ? gr_load(g + i) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      vals[e][j] *= inv_den;
      ss = fmaf(vals[e][j], vals[e][j], ss);  // (spl_finish has the same sums in the same order)
    }
  }
  const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)n + eps);
  const float* wv = weight ? weight + (weight_per_head ? (size_t)h * n : 0) : nullptr;
  T* o = out + (size_t)t * out_stride + (size_t)h * n;
#pragma unroll
  for (int e = 0; e < GROUPS; ++e) {
    const int i = V * (lane + 32 * e);
    if (i < n) {
      T res[V];
#pragma unroll
      for (int j = 0; j < V; ++j) {
        float y = vals[e][j] * inv;
        if (wv) y *= wv[i + j];
        if (g) {
          const float gv = gates[e][j];
          y *= gate_act == 2 ? gv * gr_logistic(gv) : (gate_act == 1 ? gr_logistic(gv) : gv);
        }
        res[j] = from_f32<T>(y * out_scale);
      }
      if constexpr (V == 1) {
        o[i] = res[0];
      } else if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(o + i) = make_float4(res[0], res[1], res[2], res[3]);
      } else {
        uint2 u;
        __nv_bfloat162 lo = __halves2bfloat162(res[0], res[1]), hi = __halves2bfloat162(res[2], res[3]);
        u.x = *reinterpret_cast<uint32_t*>(&lo);
        u.y = *reinterpret_cast<uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(o + i) = u;
      }
    }
  }
}

RL_API int rl_head_norm_gate(const float* x, int x_stride, int xh, const float* m, float den_eps, const float* weight, int weight_per_head,
                             float eps, const void* gate, int gate_stride, int gate_act, float out_scale, void* out, int out_stride,
                             int act_dtype, int n_rows, int H, int n, cudaStream_t stream) {
  if (n_rows <= 0 || H <= 0 || n <= 0 || !x || !out) RL_REFUSE(1, "head_norm_gate: rows=%d H=%d n=%d", n_rows, H, n);
  if (n > 32 * HN_MAX_PER_LANE) RL_REFUSE(2, "head_norm_gate: a head of %d values exceeds %d", n, 32 * HN_MAX_PER_LANE);
  if (xh < n + (m != nullptr ? 1 : 0)) RL_REFUSE(3, "head_norm_gate: head stride %d too small", xh);
  const long long pairs = (long long)n_rows * H;
  const int blocks = (int)((pairs + 3) / 4);
  const uintptr_t four = act_dtype == RL_BF16 ? 7 : 15;
  const bool wide = n % 4 == 0 && xh % 4 == 0 && x_stride % 4 == 0 && out_stride % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)out & four) == 0 &&
                    (!gate || (gate_stride % 4 == 0 && ((uintptr_t)gate & four) == 0));
#define RL_HN(T)                                                                                                                        \
  RL_LAUNCH_CHECK(rl_launch(wide ? head_norm_gate_kernel<T, 4> : head_norm_gate_kernel<T, 1>, blocks, 128, 0, stream, x, x_stride, xh, m, \
                            den_eps, weight, weight_per_head, eps, (const T*)gate, gate_stride, gate_act, out_scale, (T*)out, out_stride, \
                            n_rows, H, n))
  if (act_dtype == RL_BF16) RL_HN(bf16);
  else if (act_dtype == RL_F32) RL_HN(float);
  else
    RL_REFUSE(4, "head_norm_gate: unknown dtype %d", act_dtype);
#undef RL_HN
  return 0;
}
