// A routed feed-forward: every token is sent to `top` of E small gated feed-forwards.
//
//   moe_router   z = W_r x in 32-bit, s = softmax(z) over all experts (or s = logistic(z), each expert on its own); the
//                `top` experts with the largest s + bias are chosen (ties to the lower index), their weights are their s
//                (optionally divided by their sum plus a small constant), times a constant factor; one more row of W_r,
//                if present, gives a per-token gate sigmoid(w_g . x)
//   moe_plan     counts the (token, choice) pairs of each expert, lays them out expert after expert (`order`,
//                with the inverse `place`), and cuts each expert's range into row tiles (`tiles`) of a given height
//   moe_gemm     one kernel for all experts: a block takes one row tile (rows of ONE expert) and one column
//                tile; rows are gathered through `order`; with ACT the block computes the gate and the up
//                product together and writes act(gate) * up; without it the sums may go through relu(x)^2
//   moe_combine  out[t] = sum_j weight[t,j] * y[place[t,j]]  (+ gate[t] * shared[t]), in the order j = 0, 1, ...
//
// The router may score more choices than there are experts: those behind the experts hand the token's input on.  They have
// no rows in the plan (their place is -1), and moe_combine takes x[t] in the place of y for them.
//
// Nothing here depends on the host knowing how many tokens an expert got: grids are sized by upper bounds and
// blocks without work leave, so a step with these kernels can be captured in a CUDA graph.  Each output is one
// running 32-bit sum over ascending k, whatever the tile it lies in: a token's result does not depend on what
// else is in the batch.
#include <float.h>

#include "common.cuh"

RL_DEFINE_ERROR_TEXT()

#define MOE_TM 32  // rows of a tile: the (token, choice) pairs of one expert, 32 at a time
#define MOE_TN 64
#define MOE_TK 16

// ---------------------------------------------------------------- router
// Two kernels.  Logits: a block takes 8 tokens and 16 rows of w (four per warp), so that a row of w is read once for 8
// tokens and a token's activations once for four rows; every logit is one lane-strided sum
// followed by the warp's fixed reduction, whatever else is in the batch.  Choice: one warp per token.
// w: float32 [E (+1), d]; x in the activation type.
#define ROUTER_TOKENS 8

#define ROUTER_ROWS 4  // rows of w per warp: a token's activations are read once for four logits

template <typename T, bool VEC>
__global__ void moe_router_logits_kernel(const T* __restrict__ x, int ldx, const float* __restrict__ w, int rows, int d, int n_tokens,
                                         float* __restrict__ z) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e0 = (blockIdx.y * 4 + warp) * ROUTER_ROWS, t0 = blockIdx.x * ROUTER_TOKENS;
  if (e0 >= rows) return;
  float s[ROUTER_ROWS][ROUTER_TOKENS];
#pragma unroll
  for (int r = 0; r < ROUTER_ROWS; ++r)
#pragma unroll
    for (int i = 0; i < ROUTER_TOKENS; ++i) s[r][i] = 0.f;
  if (VEC) {  // d a multiple of 8, rows 16-byte aligned: a lane takes 8 neighbouring k per round
    for (int k = lane * 8; k < d; k += 256) {
      float wv[ROUTER_ROWS][8];
#pragma unroll
      for (int r = 0; r < ROUTER_ROWS; ++r) {
        const float* wr = w + (size_t)min(e0 + r, rows - 1) * d + k;
        load4<float>(wr, wv[r]);
        load4<float>(wr + 4, wv[r] + 4);
      }
#pragma unroll
      for (int i = 0; i < ROUTER_TOKENS; ++i)
        if (t0 + i < n_tokens) {
          float xv[8];
          load4<T>(x + (size_t)(t0 + i) * ldx + k, xv);
          load4<T>(x + (size_t)(t0 + i) * ldx + k + 4, xv + 4);
#pragma unroll
          for (int r = 0; r < ROUTER_ROWS; ++r)
#pragma unroll
            for (int u = 0; u < 8; ++u) s[r][i] += xv[u] * wv[r][u];
        }
    }
  } else {
    for (int k = lane; k < d; k += 32) {
      float wv[ROUTER_ROWS];
#pragma unroll
      for (int r = 0; r < ROUTER_ROWS; ++r) wv[r] = w[(size_t)min(e0 + r, rows - 1) * d + k];
#pragma unroll
      for (int i = 0; i < ROUTER_TOKENS; ++i)
        if (t0 + i < n_tokens) {
          const float xv = to_f32(x[(size_t)(t0 + i) * ldx + k]);
#pragma unroll
          for (int r = 0; r < ROUTER_ROWS; ++r) s[r][i] += xv * wv[r];
        }
    }
  }
#pragma unroll
  for (int r = 0; r < ROUTER_ROWS; ++r)
#pragma unroll
    for (int i = 0; i < ROUTER_TOKENS; ++i) {
      const float v = warp_sum(s[r][i]);
      if (lane == 0 && t0 + i < n_tokens && e0 + r < rows) z[(size_t)(t0 + i) * rows + e0 + r] = v;
    }
}

// Ordered as floats are, as unsigned integers (what is no number does not get here).
__device__ __forceinline__ unsigned moe_key(float v) {
  const unsigned u = __float_as_uint(v);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}

// One warp per token (four tokens per block): softmax over the E logits (or the logistic function of each), the `top` largest of
// score + bias; weights s_e (/ (sum of the chosen s + renorm_eps) if renorm) * weight_scale.  logits: `parts` partial sums
// [parts, n_tokens, rows], added up here in order.
// A lane has the experts lane + 32 i in registers (EACH of them); a round of the choice is a warp-wide maximum of keys and a minimum of the
// indices that have it, two instructions where ten shuffles were, and nothing is read back from memory: 2048 tokens, 6 of 64: 4.4 us instead of 16.
template <int EACH>
__global__ void __launch_bounds__(128)
moe_router_choose_kernel(const float* __restrict__ logits, int parts, const float* __restrict__ bias, int E, int rows, int top,
                         int renorm, int n_tokens, int* __restrict__ ids, float* __restrict__ weights,
                         float* __restrict__ gate, int logistic, float renorm_eps, float weight_scale) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * 4 + warp;
  if (t >= n_tokens) return;
  const float* lg = logits + (size_t)t * rows;
  const size_t part = (size_t)n_tokens * rows;
  float z[EACH];
  float gate_z = 0.f;
#pragma unroll
  for (int i = 0; i < EACH; ++i) z[i] = 0.f;
  constexpr int AHEAD = EACH <= 16 ? 4 : 1;  // partial sums asked for at once (four of 48 experts a lane would not fit its registers)
  for (int p0 = 0; p0 < parts; p0 += AHEAD) {
    float v[AHEAD][EACH], gv[AHEAD];
#pragma unroll
    for (int p = 0; p < AHEAD; ++p) {
      const bool in = p0 + p < parts;
#pragma unroll
      for (int i = 0; i < EACH; ++i) v[p][i] = in && lane + 32 * i < E ? __ldcg(lg + (p0 + p) * part + lane + 32 * i) : 0.f;
      gv[p] = in && rows > E ? __ldcg(lg + (p0 + p) * part + E) : 0.f;
    }
#pragma unroll
    for (int p = 0; p < AHEAD; ++p) {
#pragma unroll
      for (int i = 0; i < EACH; ++i) z[i] = p0 + p ? z[i] + v[p][i] : v[p][i];
      gate_z = p0 + p ? gate_z + gv[p] : gv[p];
    }
  }
  float mx = -INFINITY, sum = 0.f;
  if (!logistic) {
#pragma unroll
    for (int i = 0; i < EACH; ++i)
      if (lane + 32 * i < E) mx = fmaxf(mx, z[i]);
    mx = warp_max(mx);
#pragma unroll
    for (int i = 0; i < EACH; ++i)
      if (lane + 32 * i < E) {
        z[i] = expf(z[i] - mx);
        sum += z[i];
      }
    sum = warp_sum(sum);
  }
  unsigned key[EACH];
#pragma unroll
  for (int i = 0; i < EACH; ++i) {
    const int e = lane + 32 * i;
    z[i] = logistic ? 1.0f / (1.0f + expf(-z[i])) : z[i] / sum;
    // (also what is not a number: every expert stays one that can be chosen once)
    key[i] = e < E ? moe_key(fmaxf(z[i] + (bias ? bias[e] : 0.f), -FLT_MAX)) : 0u;
  }
  float chosen_sum = 0.f, mine = 0.f;  // mine: lane j keeps the j-th choice's score (top <= 32), or the last of its round of 32
  for (int j = 0; j < top; ++j) {
    unsigned best = 0;
#pragma unroll
    for (int i = 0; i < EACH; ++i) best = max(best, key[i]);
    best = __reduce_max_sync(0xffffffffu, best);
    unsigned at = 0xffffffffu;
#pragma unroll
    for (int i = EACH - 1; i >= 0; --i)
      if (key[i] == best && lane + 32 * i < E) at = lane + 32 * i;  // the lower index keeps a tie
    at = __reduce_min_sync(0xffffffffu, at);
    float score = 0.f;
#pragma unroll
    for (int i = 0; i < EACH; ++i)
      if (lane + 32 * i == (int)at) {
        score = z[i];
        key[i] = 0u;
      }
    score = __shfl_sync(0xffffffffu, score, at & 31);
    chosen_sum += score;
    if ((j & 31) == lane) {
      mine = score;
      ids[(size_t)t * top + j] = (int)at;
      if (top > 32) weights[(size_t)t * top + j] = score;
    }
  }
  if (top <= 32) {
    if (lane < top) weights[(size_t)t * top + lane] = (renorm ? mine / (chosen_sum + renorm_eps) : mine) * weight_scale;
  } else {
    for (int j = lane; j < top; j += 32) {  // (written by this very lane)
      const float w = weights[(size_t)t * top + j];
      weights[(size_t)t * top + j] = (renorm ? w / (chosen_sum + renorm_eps) : w) * weight_scale;
    }
  }
  if (rows > E && lane == 0) gate[t] = 1.0f / (1.0f + expf(-gate_z));
}

#define MOE_MAX_EXPERTS 1536  // as the former kernel's shared memory had room for
static int launch_choose(const float* logits, int parts, const float* bias, int E, int rows, int top, int renorm, int n_tokens, int* ids,
                         float* weights, float* gate, int logistic, float renorm_eps, float weight_scale, cudaStream_t stream) {
  const int blocks = (n_tokens + 3) / 4;
#define RL_CHOOSE(EACH)                                                                                                                  \
  RL_LAUNCH_CHECK(rl_launch(moe_router_choose_kernel<EACH>, blocks, 128, 0, stream, logits, parts, bias, E, rows, top, renorm, n_tokens, \
                            ids, weights, gate, logistic, renorm_eps, weight_scale))
  if (E <= 32) RL_CHOOSE(1);
  else if (E <= 64) RL_CHOOSE(2);
  else if (E <= 128) RL_CHOOSE(4);
  else if (E <= 256) RL_CHOOSE(8);
  else if (E <= 512) RL_CHOOSE(16);
  else if (E <= 768) RL_CHOOSE(24);
  else if (E <= 1024) RL_CHOOSE(32);
  else RL_CHOOSE(48);
#undef RL_CHOOSE
  return 0;
}

// logits: float32 scratch of n_tokens * (E + has_gate) values.
RL_API int rl_moe_router(const void* x, int ldx, int dtype, const float* w, const float* bias, int n_tokens, int E, int d,
                         int top, int renorm, int has_gate, float* logits, int* ids, float* weights, float* gate, int logistic,
                         float renorm_eps, float weight_scale, cudaStream_t stream) {
  if (n_tokens <= 0 || E <= 0 || d <= 0 || top <= 0 || top > E) RL_REFUSE(1, "moe_router: T=%d E=%d d=%d top=%d", n_tokens, E, d, top);
  if (has_gate && gate == nullptr) RL_REFUSE(2, "moe_router: a gate row but nowhere to write the gate");
  if (E > MOE_MAX_EXPERTS) RL_REFUSE(3, "moe_router: %d experts exceed %d", E, MOE_MAX_EXPERTS);
  const int rows = E + (has_gate ? 1 : 0);
  dim3 grid((n_tokens + ROUTER_TOKENS - 1) / ROUTER_TOKENS, (rows + 4 * ROUTER_ROWS - 1) / (4 * ROUTER_ROWS));
  if (grid.y > 65535) RL_REFUSE(5, "moe_router: %d experts exceed the grid", E);
  // (which of the two loops runs depends on sizes and addresses only, never on the batch: a token's logits keep their bits)
  const bool vec = d % 8 == 0 && ldx % 8 == 0 && ((uintptr_t)x % 16 == 0) && ((uintptr_t)w % 16 == 0);
  if (dtype == RL_BF16 && vec)
    RL_LAUNCH_CHECK(rl_launch<false>(moe_router_logits_kernel<bf16, true>, grid, 128, 0, stream, (const bf16*)x, ldx, w, rows, d, n_tokens, logits));
  else if (dtype == RL_BF16)
    RL_LAUNCH_CHECK(rl_launch<false>(moe_router_logits_kernel<bf16, false>, grid, 128, 0, stream, (const bf16*)x, ldx, w, rows, d, n_tokens, logits));
  else if (dtype == RL_F32 && vec)
    RL_LAUNCH_CHECK(rl_launch<false>(moe_router_logits_kernel<float, true>, grid, 128, 0, stream, (const float*)x, ldx, w, rows, d, n_tokens, logits));
  else if (dtype == RL_F32)
    RL_LAUNCH_CHECK(rl_launch<false>(moe_router_logits_kernel<float, false>, grid, 128, 0, stream, (const float*)x, ldx, w, rows, d, n_tokens, logits));
  else
    RL_REFUSE(4, "moe_router: unknown dtype %d", dtype);
  return launch_choose(logits, 1, bias, E, rows, top, renorm, n_tokens, ids, weights, gate, logistic, renorm_eps, weight_scale, stream);
}

// The choice alone, from logits that another product made (float32 [parts, n_tokens, E + has_gate], partial sums).
RL_API int rl_moe_choose(const float* logits, int parts, const float* bias, int n_tokens, int E, int top, int renorm, int has_gate, int* ids, float* weights,
                         float* gate, int logistic, float renorm_eps, float weight_scale, cudaStream_t stream) {
  if (n_tokens <= 0 || E <= 0 || top <= 0 || top > E) RL_REFUSE(1, "moe_choose: T=%d E=%d top=%d", n_tokens, E, top);
  if (has_gate && gate == nullptr) RL_REFUSE(2, "moe_choose: a gate column but nowhere to write the gate");
  if (E > MOE_MAX_EXPERTS) RL_REFUSE(3, "moe_choose: %d experts exceed %d", E, MOE_MAX_EXPERTS);
  if (parts <= 0) RL_REFUSE(4, "moe_choose: %d partial sums", parts);
  return launch_choose(logits, parts, bias, E, E + (has_gate ? 1 : 0), top, renorm, n_tokens, ids, weights, gate, logistic, renorm_eps, weight_scale, stream);
}

// ---------------------------------------------------------------- plan
// ids[n] (n = T * top pairs) -> order[n] (pairs laid out expert after expert, each expert's pairs in ascending
// pair index), place[pair] (its row in that layout), tiles[1 + 3 * max_tiles]: the number of tiles, then
// (expert, first row, rows) per tile.  One block per expert: every block counts all experts' pairs in shared memory
// (it needs the counts of the experts before its own for its first row and its first tile), then lays out its own
// expert's pairs, each thread a contiguous piece of the pairs so that their order is kept.
// `always` further matrices, numbers E and up, take every token (a shared expert in pieces of the others' size): their rows come behind the n
// of the pairs, row n + j T + t is token t's of the j-th (order: its first pair).  Their tiles stand between the others', evenly: blocks that
// wait for an expert's weights are then beside blocks whose matrix is in L2 and whose rows are many.
#define PLAN_THREADS 512

// where the i-th of `few` tiles stands among `all`, and how many of the few stand before place p
__device__ __forceinline__ int plan_place(int i, int few, int all) { return (int)(((long long)i * all) / few); }
__device__ __forceinline__ int plan_before(int p, int few, int all) {  // the least i with plan_place(i) >= p
  return (int)(((long long)p * few + all - 1) / all);
}

template <bool MANY>  // pairs, eight or more a thread, whose ids are 16-byte aligned
__global__ void __launch_bounds__(PLAN_THREADS)
moe_plan_kernel(const int* __restrict__ ids, int n, int E, int* __restrict__ order, int* __restrict__ place,
                int* __restrict__ tiles, int tile_rows, int always, int top) {
  extern __shared__ int cnt[];  // E counts
  __shared__ int scan[PLAN_THREADS / 32], sums[3];
  pdl_trigger();
  pdl_wait();
  const int e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < E; i += PLAN_THREADS) cnt[i] = 0;
  if (tid < 3) sums[tid] = 0;
  __syncthreads();
  // A thread has neighbouring pairs, eight of which are asked for at once (one after the other the trips to L2 were most of the kernel), of MANY by 16
  // bytes: 2048 tokens of 6 12.1 us instead of 14.3.
  int per = (n + PLAN_THREADS - 1) / PLAN_THREADS;
  if (MANY) per = (per + 7) & ~7;
  const int lo = min(n, tid * per), hi = min(n, lo + per);
  auto load = [&](int i0, int (&id)[8], int none) {
    if (MANY && i0 + 7 < hi) {
      const int4 v = __ldcg(reinterpret_cast<const int4*>(ids + i0)), w = __ldcg(reinterpret_cast<const int4*>(ids + i0 + 4));
      id[0] = v.x, id[1] = v.y, id[2] = v.z, id[3] = v.w, id[4] = w.x, id[5] = w.y, id[6] = w.z, id[7] = w.w;
      return;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) id[u] = i0 + u < hi ? __ldcg(ids + i0 + u) : none;
  };
  int mine = 0;
  for (int i0 = lo; i0 < hi; i0 += 8) {
    int id[8];
    load(i0, id, 0);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + u < hi) {
        if (id[u] < E) atomicAdd(&cnt[id[u]], 1);
        else if (e == 0) place[i0 + u] = -1;  // (no expert of the plan: it has no row)
        mine += id[u] == e;
      }
  }
  int before = mine;  // of this warp's threads up to this one
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += v;
  }
  if (lane == 31) scan[warp] = before;
  __syncthreads();
  for (int k = tid; k < E; k += PLAN_THREADS) {  // rows and tiles of the experts before this one, tiles of all
    const int c = cnt[k], nt = (c + tile_rows - 1) / tile_rows;
    if (k < e) {
      atomicAdd(&sums[0], c);
      atomicAdd(&sums[1], nt);
    }
    atomicAdd(&sums[2], nt);
  }
  __syncthreads();
  const int T = n / top, per_always = (T + tile_rows - 1) / tile_rows, few = always * per_always, all = sums[2] + few;
  if (e == 0 && tid == 0) tiles[0] = all;
  int first_row, first_tile, c;
  if (e < E) {
    first_row = sums[0];
    first_tile = sums[1];
    c = cnt[e];
    int r = first_row + before - mine;
    for (int w = 0; w < warp; ++w) r += scan[w];
    for (int i0 = lo; i0 < hi && mine > 0; i0 += 8) {
      int id[8];
      load(i0, id, -1);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i0 + u < hi && id[u] == e) {
          order[r] = i0 + u;
          place[i0 + u] = r;
          ++r;
          --mine;
        }
    }
  } else {
    first_row = n + (e - E) * T;
    first_tile = (e - E) * per_always;
    c = T;
    for (int t = tid; t < T; t += PLAN_THREADS) order[first_row + t] = t * top;
  }
  // As few tiles as hold the expert's rows.  Where the products take tiles of any multiple of 16 rows (the heights from 128 on) they
  // are equally high: 300 rows in two tiles of 160 and 140 instead of 256 and 44 (no last tile is empty: the others hold at most
  // tile_rows each).
  const int n_tiles = (c + tile_rows - 1) / tile_rows;
  int high = tile_rows;
  if (tile_rows >= 128 && n_tiles > 0) high = min(tile_rows, ((c + n_tiles - 1) / n_tiles + 15) & ~15);
  for (int k = tid; k < n_tiles; k += PLAN_THREADS) {
    int at = first_tile + k;
    if (e >= E) {
      at = plan_place(at, few, all);
    } else if (few > 0) {
      // the at-th place that none of the few has: places before p that are free are p - plan_before(p); find the first p with at + 1 of them
      int lo_p = at, hi_p = at + few;
      while (lo_p < hi_p) {
        const int p = (lo_p + hi_p) >> 1;
        if (p + 1 - plan_before(p + 1, few, all) >= at + 1) hi_p = p;
        else lo_p = p + 1;
      }
      at = lo_p;
    }
    int* t = tiles + 1 + 3 * at;
    t[0] = e;
    t[1] = first_row + k * high;
    t[2] = min(high, c - k * high);
  }
}

// ---------------------------------------------------------------- experts chosen by a table instead of a router
// ids[t][j] = table[token[t]][j], every chosen expert with the weight 1 / top.
__global__ void moe_table_lookup_kernel(const int* __restrict__ tokens, const int* __restrict__ table, int top, int n, int E,
                                        int* __restrict__ ids, float* __restrict__ weights) {
  pdl_trigger();
  pdl_wait();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n * top) return;
  const int t = idx / top, j = idx - t * top;
  const int e = table[(size_t)tokens[t] * top + j];
  ids[idx] = min(max(e, 0), E - 1);  // (the loader has checked the table; a stray id must still not index outside the weights)
  weights[idx] = 1.0f / (float)top;
}

RL_API int rl_moe_table_lookup(const int* tokens, const int* table, int top, int n_tokens, int E, int* ids, float* weights, cudaStream_t stream) {
  if (n_tokens <= 0 || top <= 0 || E <= 0) RL_REFUSE(1, "moe_table_lookup: T=%d top=%d E=%d", n_tokens, top, E);
  const int total = n_tokens * top;
  RL_LAUNCH_CHECK(rl_launch(moe_table_lookup_kernel, (total + 255) / 256, 256, 0, stream, tokens, table, top, n_tokens, E, ids, weights));
  return 0;
}

RL_API int rl_moe_tile_rows() { return MOE_TM; }

RL_API int rl_moe_plan(const int* ids, int n, int E, int* order, int* place, int* tiles, int tile_rows, int always, int top, cudaStream_t stream) {
  if (n <= 0 || E <= 0 || tile_rows <= 0 || always < 0 || top <= 0 || n % top) RL_REFUSE(1, "moe_plan: n=%d E=%d tile_rows=%d always=%d top=%d", n, E, tile_rows, always, top);
  const size_t smem = (size_t)E * sizeof(int);
  if (smem > 40 * 1024) RL_REFUSE(2, "moe_plan: %d experts exceed the kernel's shared memory", E);
  const bool many = n > 7 * PLAN_THREADS && ((uintptr_t)ids & 15) == 0;
  RL_LAUNCH_CHECK(rl_launch(many ? moe_plan_kernel<true> : moe_plan_kernel<false>, E + always, PLAN_THREADS, smem, stream, ids, n, E, order, place, tiles, tile_rows, always, top));
  return 0;
}

// ---------------------------------------------------------------- all experts' products in one launch
// Row r of the layout belongs to pair order[r]; its input row is x[order[r] / gather_div] when `order` is given
// (the token's activations), else x[r].  w: [E, N, K]; with ACT also w2: [E, N, K] and out = gated_act(x w^T, x w2^T): silu(g) * u,
// or with a limit the clamped form (common.cuh).
// blockIdx.y walks the tiles of the plan; a block beyond the plan's count leaves.
template <typename TA, typename TO, bool ACT>
__global__ void __launch_bounds__(256)
moe_gemm_kernel(const TA* __restrict__ x, int ldx, const int* __restrict__ order, int gather_div, const TA* __restrict__ w,
                const TA* __restrict__ w2, TO* __restrict__ out, int ldo, const int* __restrict__ tiles, int N, int K, float act_alpha,
                float act_limit) {
  __shared__ float xs[MOE_TK][MOE_TM + 4];
  __shared__ float ws[MOE_TK][MOE_TN + 4];
  __shared__ float ws2[ACT ? MOE_TK : 1][MOE_TN + 4];
  __shared__ int src[MOE_TM];
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.y >= tiles[0]) return;
  const int e = tiles[1 + 3 * blockIdx.y], r0 = tiles[2 + 3 * blockIdx.y], rows = tiles[3 + 3 * blockIdx.y];
  const int tid = threadIdx.x, n0 = blockIdx.x * MOE_TN;
  const int ty = tid / 16, tx = tid % 16;  // 16 x 16 threads: 2 rows x 4 columns each
  if (tid < MOE_TM) src[tid] = tid < rows ? (order ? order[r0 + tid] / gather_div : r0 + tid) : -1;
  __syncthreads();
  const TA* we = w + (size_t)e * N * K;
  const TA* we2 = ACT ? w2 + (size_t)e * N * K : nullptr;
  float acc[2][4], acc2[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = acc2[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += MOE_TK) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int idx = tid + i * 256;
      const int r = idx / MOE_TK, c = idx % MOE_TK;
      const int k = k0 + c;
      xs[c][r] = (src[r] >= 0 && k < K) ? to_f32(x[(size_t)src[r] * ldx + k]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256;
      const int r = idx / MOE_TK, c = idx % MOE_TK;
      const int k = k0 + c;
      const bool in = n0 + r < N && k < K;
      ws[c][r] = in ? to_f32(we[(size_t)(n0 + r) * K + k]) : 0.f;
      if (ACT) ws2[c][r] = in ? to_f32(we2[(size_t)(n0 + r) * K + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < MOE_TK; ++c) {
      float a[2], b[4], b2[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = xs[c][ty * 2 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b[j] = ws[c][tx * 4 + j];
        if (ACT) b2[j] = ws2[c][tx * 4 + j];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
          if (ACT) acc2[i][j] = fmaf(a[i], b2[j], acc2[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = ty * 2 + i;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (ACT) v = gated_act(v, acc2[i][j], act_alpha, act_limit);
      else v = unary_post(v, act_limit);
      out[(size_t)(r0 + r) * ldo + n] = from_f32<TO>(v);
    }
  }
}

// (the plan's tiles must be MOE_TM rows high: `rl_moe_tile_rows`)
RL_API int rl_moe_gemm(const void* x, int ldx, int dtype, const int* order, int gather_div, const void* w, const void* w2,
                       void* out, int out_dtype, int ldo, const int* tiles, int max_tiles, int N, int K, float act_alpha, float act_limit,
                       cudaStream_t stream) {
  if (max_tiles <= 0 || N <= 0 || K <= 0 || gather_div <= 0) RL_REFUSE(1, "moe_gemm: tiles=%d N=%d K=%d div=%d", max_tiles, N, K, gather_div);
  if (max_tiles > 65535) RL_REFUSE(2, "moe_gemm: %d row tiles exceed the grid", max_tiles);
  dim3 grid((N + MOE_TN - 1) / MOE_TN, max_tiles);
#define RL_MG(TA, TO, ACT)                                                                                                  \
  RL_LAUNCH_CHECK(rl_launch<false>(moe_gemm_kernel<TA, TO, ACT>, grid, 256, 0, stream, (const TA*)x, ldx, order, gather_div, \
                                   (const TA*)w, (const TA*)w2, (TO*)out, ldo, tiles, N, K, act_alpha, act_limit))
  if (dtype == RL_BF16 && out_dtype == RL_BF16 && w2) RL_MG(bf16, bf16, true);
  else if (dtype == RL_BF16 && out_dtype == RL_BF16) RL_MG(bf16, bf16, false);
  else if (dtype == RL_BF16 && out_dtype == RL_F32 && !w2) RL_MG(bf16, float, false);
  else if (dtype == RL_F32 && out_dtype == RL_F32 && w2) RL_MG(float, float, true);
  else if (dtype == RL_F32 && out_dtype == RL_F32) RL_MG(float, float, false);
  else RL_REFUSE(3, "moe_gemm: unsupported types in=%d out=%d act=%d", dtype, out_dtype, w2 != nullptr);
#undef RL_MG
  return 0;
}

// ---------------------------------------------------------------- weighted sum of a token's experts
// out[t, :] = sum_j weights[t, j] * y[place[t * top + j], :]  (+ gate[t] * shared[t, :]); y is float32.  A negative place takes
// x[t, :], the experts' input (of type TS, like `shared`), in the place of y.  The rows of `always` further matrices (see the plan) are
// y[T top + j T + t, :]: their sum is a shared expert's result, and like the one that comes as `shared` from products of its own it is
// rounded to bfloat16 before it counts gate[t] (1 without a gate) times, so that a token's result does not depend on which way it went.
template <typename TS, typename TO>
__global__ void moe_combine_kernel(const float* __restrict__ y, const int* __restrict__ place, const float* __restrict__ weights,
                                   int top, const TS* __restrict__ shared, const float* __restrict__ gate, TO* __restrict__ out, int d,
                                   const TS* __restrict__ x, int ldx, int always) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    float v = 0.f;
    for (int j = 0; j < top; ++j) {
      const int p = place[(size_t)t * top + j];
      v += weights[(size_t)t * top + j] * (p >= 0 ? y[(size_t)p * d + i] : x != nullptr ? to_f32(x[(size_t)t * ldx + i]) : 0.f);
    }
    if (shared) v += (gate ? gate[t] : 1.f) * to_f32(shared[(size_t)t * d + i]);
    if (always > 0) {
      float s = 0.f;
      for (int j = 0; j < always; ++j) s += y[((size_t)gridDim.x * (top + j) + t) * d + i];
      v += (gate ? gate[t] : 1.f) * to_f32(__float2bfloat16_rn(s));
    }
    out[(size_t)t * d + i] = from_f32<TO>(v);
  }
}

// The same sums, four neighbouring columns a thread and everything a thread needs of eight choices in flight at once.
// With rows of matrices that take every token (OWN) the first of those are asked for before the choices': where they are is known.
#define COMBINE_AHEAD 8
#define COMBINE_OWN 2
template <typename TS, typename TO, bool OWN>
__global__ void __launch_bounds__(256)
moe_combine_vec_kernel(const float* __restrict__ y, const int* __restrict__ place, const float* __restrict__ weights, int top,
                       const TS* __restrict__ shared, const float* __restrict__ gate, TO* __restrict__ out, int d,
                       const TS* __restrict__ x, int ldx, int always) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, i = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (i >= d) return;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  float ahead[COMBINE_OWN][4];
  const float* own_row = y + ((size_t)gridDim.x * top + t) * d + i;
  const size_t own_step = (size_t)gridDim.x * d;
  if constexpr (OWN) {
#pragma unroll
    for (int j = 0; j < COMBINE_OWN; ++j) {
      ahead[j][0] = ahead[j][1] = ahead[j][2] = ahead[j][3] = 0.f;
      if (j < always) load4_g<float>(own_row + j * own_step, ahead[j]);
    }
  }
  for (int j0 = 0; j0 < top; j0 += COMBINE_AHEAD) {
    int p[COMBINE_AHEAD];
    float w[COMBINE_AHEAD], f[COMBINE_AHEAD][4];
#pragma unroll
    for (int u = 0; u < COMBINE_AHEAD; ++u) {
      const bool in = j0 + u < top;
      p[u] = in ? __ldcg(place + (size_t)t * top + j0 + u) : -1;
      w[u] = in ? __ldcg(weights + (size_t)t * top + j0 + u) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < COMBINE_AHEAD; ++u) {
      if (j0 + u >= top || (p[u] < 0 && x == nullptr)) f[u][0] = f[u][1] = f[u][2] = f[u][3] = 0.f;
      else if (p[u] >= 0) load4_g<float>(y + (size_t)p[u] * d + i, f[u]);
      else load4_g<TS>(x + (size_t)t * ldx + i, f[u]);
    }
#pragma unroll
    for (int u = 0; u < COMBINE_AHEAD; ++u)
      if (j0 + u < top)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] += w[u] * f[u][e];
  }
  if (shared || OWN) {
    const float g = gate ? __ldcg(gate + t) : 1.f;
    if (shared) {
      float s[4];
      load4_g<TS>(shared + (size_t)t * d + i, s);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] += g * s[e];
    }
    if constexpr (OWN) {
      float own[4] = {ahead[0][0], ahead[0][1], ahead[0][2], ahead[0][3]};
#pragma unroll
      for (int j = 1; j < COMBINE_OWN; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) own[e] += ahead[j][e];
      for (int j = COMBINE_OWN; j < always; ++j) {
        float f[4];
        load4_g<float>(own_row + j * own_step, f);
#pragma unroll
        for (int e = 0; e < 4; ++e) own[e] += f[e];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] += g * to_f32(__float2bfloat16_rn(own[e]));
    }
  }
  store4<TO>(out + (size_t)t * d + i, v);
}

RL_API int rl_moe_combine(const float* y, const int* place, const float* weights, int top, const void* shared, int shared_dtype,
                          const float* gate, void* out, int out_dtype, int n_tokens, int d, const void* x, int x_dtype, int ldx, int always,
                          cudaStream_t stream) {
  if (n_tokens <= 0 || d <= 0 || top <= 0 || always < 0) RL_REFUSE(1, "moe_combine: T=%d d=%d top=%d always=%d", n_tokens, d, top, always);
  if ((long long)n_tokens * (top + always) > 0x7fffffffLL) RL_REFUSE(4, "moe_combine: %d tokens of %d choices are too many", n_tokens, top + always);
  if (shared == nullptr && x != nullptr) shared_dtype = x_dtype;
  if (x != nullptr && shared_dtype != x_dtype) RL_REFUSE(3, "moe_combine: shared result of type %d beside an input of type %d", shared_dtype, x_dtype);
  // (which kernel runs depends on sizes and addresses only; both add in the same order)
  const bool vec = d % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)y | (uintptr_t)shared | (uintptr_t)out | (uintptr_t)x) & 15) == 0;
  dim3 grid(n_tokens, (d / 4 + 255) / 256);
#define RL_MC(TS, TO)                                                                                                          \
  if (vec)                                                                                                                     \
    RL_LAUNCH_CHECK(rl_launch(always > 0 ? moe_combine_vec_kernel<TS, TO, true> : moe_combine_vec_kernel<TS, TO, false>, grid, 256, 0, stream, y, place, weights, top, (const TS*)shared, gate, \
                              (TO*)out, d, (const TS*)x, ldx, always));                                                        \
  else                                                                                                                         \
  RL_LAUNCH_CHECK(rl_launch<false>(moe_combine_kernel<TS, TO>, n_tokens, 256, 0, stream, y, place, weights, top, (const TS*)shared, \
                                   gate, (TO*)out, d, (const TS*)x, ldx, always))
  if (shared_dtype == RL_BF16 && out_dtype == RL_F32) { RL_MC(bf16, float); }
  else if (shared_dtype == RL_F32 && out_dtype == RL_F32) { RL_MC(float, float); }
  else if (shared_dtype == RL_BF16 && out_dtype == RL_BF16) { RL_MC(bf16, bf16); }
  else RL_REFUSE(2, "moe_combine: unsupported types shared=%d out=%d", shared_dtype, out_dtype);
#undef RL_MC
  return 0;
}
