// Many products with matrices of their own in one launch, bfloat16 on the 5th-generation tensor cores (tcgen05, 32-bit sums in
// tensor memory):
//
//   moe_gemm_tc     the products of a routed feed-forward.  A group is a row tile of the plan that `moe_plan` left on the device:
//                   up to NT rows of ONE expert, gathered through `order`.  With two matrices the kernel computes the gate and the
//                   up product together and writes gated_act(gate, up); with one the sums may go through relu(x)^2 (`unary_post`).
//   head_linear_tc  out[t, h, :] = W[h] x[t, h, :] for every head h, optionally times sigmoid(gate[t, h, :]).  A group is a head
//                   and up to NT tokens.
//
// The weights are the M side of the tensor core's tile (128 features, a lane of tensor memory each) and the rows the N side, whose
// width is any multiple of 16: an expert with 190 rows costs 192 columns and not two tiles of 128 rows, and its matrix is read
// once.  What bounds the kernel is that reading: every expert's matrices come from HBM once (64 experts of 1408 x 2048 and
// 2048 x 1408: 1.1 GB), so the copies of weights run ahead through a ring that holds 64 KB of them (row tiles of 256) to 160 KB
// (of 32) per SM.
//
// Persistent, one block per SM; a unit of work is a group and 128 features (gated: 64 features of each matrix, stacked in one
// tile).  Per 64-wide slice of k:
//   warp 0      (one lane) TMA: two boxes of 64 rows x 64 k of weights, 128-byte swizzled;
//   warps 10-13 (one lane each, every fourth slice) TMA: the rows, four named ones a copy (tile::gather4), or boxes of neighbouring
//               ones; k that does not exist arrives as zeros, rows past a group's last are computed and not stored;
//   warp 1      (one lane) tcgen05.mma 128 x n x 16, four per slice, and the commit that hands the stage back.  The next stage is
//               asked for before the four are issued: with n below 256 a slice's products take less time than the answer;
//   warps 2-9   a finished accumulator, read with tcgen05.ld while the other half of tensor memory fills: a warp has 32 features, so
//               a row of the output is one store of 32 neighbouring numbers.  For a gate/up tile the warps that hold a feature's
//               gate and its up sums trade halves through shared memory.
// k, the row strides and the matrices' rows must be multiples of 8 elements and 16-byte aligned; the plain kernels take the rest.
// Every wait on an mbarrier is bounded (tc_common.cuh): on expiry a code goes to status[0] and the block drains.
//
// Measured, mma.sync tiles of 128 x 64 (32 x 64 for few rows) on a two-stage ring before / this kernel after:
//   64 experts of 1408 x 2048, 2048 tokens x 6    gate and up 566 / 195 us (the rows' gather included), down 330 / 96 us
//   32 experts of 2048 x 4096, 1400 tokens x 4    786 / 237 us, 462 / 120 us (790 TFLOP/s)
//   the same, 96 tokens                           213 / 170 us, 104 / 87 us (6.2 TB/s of weights)
//   16 heads, 2048 tokens, 512 x 128 and 128 x 512 a head    50.6 / 15.8 us, 27.2 / 9.3 us
// The gate's activation keeps the exponential and the division of 32 bits: the hardware's approximations (`gated_act_fast`) were worth 1 % of a
// sublayer of 64 experts over 2048 tokens and 0.3 % of one of 32 over 96, and gave zero for gates below -87.
// Without the division's branch (common.cuh) 64 experts of 1408 x 2048 over 2048 tokens take 176 us for gate and up instead of 178, and 176
// instead of 209 where the gates are so large that the division leaves its short way.
// Rings of their own for weights and rows: with 7, 6 or 5 stages of weights beside 4 of rows equal, 3 of rows 10 % and 2 of rows 45 % slower, 5 of
// rows (192 high, which a plan of 256 does not fit) 3 % faster: what an SM waits for is its share of what L2 sends, not the weights from HBM.
// What did not help: asking the weights into L2 four to sixteen slices ahead (equal or up to 5 % slower), the rows by cp.async from
// four warps (137 us for the second product where boxes of 64 neighbouring rows take 97).  With one warp per quarter of tensor
// memory the way out bounded every unit (192 rows: 8 us plain, 18 us gated; two warps: 3.3 and 7.2).
#include "tc_common.cuh"

RL_DEFINE_ERROR_TEXT()

#define BK 64
#define FEATURES 128                       // rows of a weight tile
#define A_BYTES (FEATURES * BK * 2)
#define RESULT_WARPS 8                     // two for each quarter of tensor memory's lanes
#define GATHER_WARPS 4                     // a power of two
#define FIRST_GATHER (2 + RESULT_WARPS)
#define NUM_THREADS ((FIRST_GATHER + GATHER_WARPS) * 32)
#define MAX_STAGES 10
#define LISTED_TILES 512                   // groups whose description is kept in shared memory
#define TRADE_BYTES (4 * 2 * 2 * 8 * 32 * 4)  // [pair of warps][turn][direction][8 rows][32 features]

enum { PLAIN = 0, GATED = 1, SIGMOID = 2 };

// Four rows of 64 k named one by one, 512 bytes; 128-byte swizzled by the shared-memory address like a box of rows.
__device__ __forceinline__ void tma_gather4_s(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int4 rows) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(rows.x), "r"(rows.y), "r"(rows.z), "r"(rows.w)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_s(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

template <int NT>
struct Shape {
  static constexpr int STAGE_BYTES = A_BYTES + NT * BK * 2;
  static constexpr int STAGES = NT == 256 ? 4 : NT == 128 ? 6 : 10;
  static constexpr int BOX_ROWS = NT == 32 ? 32 : 64;  // of a copy of neighbouring rows
  static constexpr int TMEM_COLS = 2 * NT;  // two accumulators
  static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + TRADE_BYTES + GATHER_WARPS * NT * 4 + LISTED_TILES * 12;
  static_assert(STAGES <= MAX_STAGES && SMEM_BYTES <= 227 * 1024 && (STAGE_BYTES & 1023) == 0, "the ring must fit");
};

struct Groups {
  const bf16* x;       // rows: x + row * ldx (+ head * xh), x_rows of them
  long long ldx, xh;
  int x_rows;
  const int* order;    // the plan's row r is row order[r] / gather_div of x (null: row r)
  int gather_div;
  const int* tiles;    // the plan: [0] groups, then (expert, first row, rows) of each; null: heads
  int heads, M;        // heads: groups of up to NT of M tokens, head after head
  const int* held;     // heads: null, or how many rows each of M / seq_rows runs of `seq_rows` rows holds (rounded up to 64; the rest is left out)
  int seq_rows;
  long long ldo, oh;
  const bf16* gate;    // SIGMOID
  long long ldg, gh;
  int N, K;
  int matrices;        // matrices of w
  int piece_first;     // the dimensions of those beside them go by their strides: [feature][piece][k] instead of [piece][feature][k]
  int shift;           // where in a row of theirs the second half of a tile begins: behind the first matrix's K numbers, or 0
  float act_alpha, act_limit;
};

// Matrices that take every token (a shared expert in pieces of the others' size), where they lie: feature n of the j-th at w + j * piece +
// n * row, K numbers (the others' are described to TMA in the same way).  So rows of gate and up that alternate and columns of one wide
// matrix serve as they are, and no copy beside the others is held.
struct Always {
  const bf16 *w, *w2;
  long long row, piece;
  int n;
};

// How TMA finds the weights: the matrices of w (and w2), and with MORE those that take every token, the plan's groups of higher numbers.
template <bool MORE>
struct WeightMaps {
  CUtensorMap w, w2;
};
template <>
struct WeightMaps<true> {
  CUtensorMap w, w2, s, s2;
};

template <typename TO, int EPI, int NT, bool MORE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
grouped_gemm_tc_kernel(const __grid_constant__ WeightMaps<MORE> maps, const __grid_constant__ CUtensorMap map_x, TO* __restrict__ out,
                       const Groups g, int* __restrict__ status, int test_role, uint32_t test_ns) {
  using SH = Shape<NT>;
  constexpr int STAGES = SH::STAGES, UNIT_N = EPI == GATED ? FEATURES / 2 : FEATURES;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  float* trade = reinterpret_cast<float*>(stages + (size_t)STAGES * SH::STAGE_BYTES);
  int* row_ids = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(trade) + TRADE_BYTES);  // [gathering warp][NT]
  int* listed = row_ids + GATHER_WARPS * NT;
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_full[2], acc_empty[2], drain_bar;
  __shared__ uint32_t tmem_slot, weights_asked, rows_asked[GATHER_WARPS];
  __shared__ int abort_flag, go[2];
  const WaitCtl ctl = {&abort_flag, test_role, test_ns};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 2);  // the weights' bytes, the rows' warp
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], RESULT_WARPS);
    }
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_slot, SH::TMEM_COLS);
  tc_fence_before();
  pdl_trigger();
  pdl_wait();  // the plan, the rows: other kernels' output
  const int blocks_n = (g.N + UNIT_N - 1) / UNIT_N, per_run = g.held != nullptr ? (g.seq_rows + NT - 1) / NT : 0;
  const int per_head = g.held != nullptr ? g.M / g.seq_rows * per_run : (g.M + NT - 1) / NT;
  const int n_groups = g.tiles != nullptr ? __ldcg(g.tiles) : g.heads * per_head;
  if (g.tiles != nullptr)
    for (int i = threadIdx.x; i < 3 * min(n_groups, LISTED_TILES); i += NUM_THREADS) listed[i] = __ldcg(g.tiles + 1 + i);
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const int n_units = n_groups * blocks_n, n_k = (g.K + BK - 1) / BK;
  // the group of a unit: its matrix, its first row and how many (none, of a run that holds fewer: every role passes over the unit)
  auto group = [&](int unit, int& e, int& r0, int& rows) {
    const int t = unit / blocks_n;
    if (g.tiles == nullptr) {
      e = t / per_head;
      if (g.held == nullptr) {
        r0 = (t - e * per_head) * NT;
        rows = min(NT, g.M - r0);
      } else {
        const int run = (t - e * per_head) / per_run, at = (t - e * per_head - run * per_run) * NT;
        r0 = run * g.seq_rows + at;
        rows = min(NT, min(g.seq_rows, (__ldcg(g.held + run) + 63) & ~63) - at);
      }
    } else if (t < LISTED_TILES) {
      e = listed[3 * t];
      r0 = listed[3 * t + 1];
      rows = listed[3 * t + 2];
    } else {
      e = __ldcg(g.tiles + 1 + 3 * t);
      r0 = __ldcg(g.tiles + 2 + 3 * t);
      rows = __ldcg(g.tiles + 3 + 3 * t);
    }
  };
  const uint32_t stage0 = smem_u32(stages), full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);

  if (warp == 0) {
    // ---------------- weights
    if (lane == 0) {
      uint32_t it = 0, s = 0, parity = 1, dst = stage0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
        int e, r0, rows;
        group(unit, e, r0, rows);
        if (rows <= 0) continue;
        const CUtensorMap *from = &maps.w, *from2 = &maps.w2;
        const int row = (unit % blocks_n) * UNIT_N, row2 = EPI == GATED ? row : row + FEATURES / 2;
        int y = row, z = e, y2 = row2, z2 = e, shift = 0;
        if constexpr (MORE) {
          if (e >= g.matrices) {
            const int piece = e - g.matrices;
            from = &maps.s, from2 = &maps.s2;
            y = g.piece_first ? piece : row, z = g.piece_first ? row : piece;
            y2 = g.piece_first ? piece : row2, z2 = g.piece_first ? row2 : piece;
            shift = g.shift;
          }
        }
        for (int kb = 0; kb < n_k; ++kb, ++it) {
          if (it >= STAGES && !mbar_wait_role(&empty_bar[s], parity, ctl, 61)) {
            give_up_code(status, 61);
            abort_flag = 1;
            ok = false;
            break;
          }
          mbar_expect_tx_s(full0 + 8 * s, A_BYTES);
          tma_load_3d_s(dst, from, full0 + 8 * s, kb * BK, y, z);
          tma_load_3d_s(dst + A_BYTES / 2, from2, full0 + 8 * s, kb * BK + shift, y2, z2);
          dst += SH::STAGE_BYTES;
          if (++s == STAGES) {
            s = 0;
            dst = stage0;
            parity ^= 1;
          }
        }
      }
      weights_asked = it;
    }
  } else if (warp == 1) {
    // ---------------- tensor-core issuer
    if (lane == 0) {
      const uint64_t a_desc0 = make_smem_desc(stage0), b_desc0 = make_smem_desc(stage0 + A_BYTES);
      uint64_t stage_off = 0;
      uint32_t s = 0, phase = 0, ready = 0;
      bool ok = true;
      int local = 0;
      for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
        int e, r0, rows;
        group(unit, e, r0, rows);
        if (rows <= 0) continue;
        const uint32_t idesc = make_idesc(FEATURES, (rows + 15) & ~15);
        const int acc = local & 1;
        const uint32_t use = local >> 1;
        if (use > 0 && !mbar_wait_role(&acc_empty[acc], (use - 1) & 1, ctl, 64)) {
          give_up_code(status, 64);
          abort_flag = 1;
          ok = false;
          break;
        }
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * NT);
        for (int kb = 0; kb < n_k; ++kb) {
          // (A yes to the question that the slice before asked IS the wait: mbarrier.test_wait and try_wait answer for the same phase, with the
          // same visibility, and the phase cannot move on before this slice is committed.  720 000 launches in decode and mixed steps of two
          // models: no give-up.  With a wait in front of every slice all the same, 64 experts over 2048 tokens took 488 us and not 482, 32 over
          // 96 tokens 366 and not 351.)
          if (!ready && !mbar_wait_role(&full_bar[s], phase, ctl, 62)) {
            give_up_code(status, 62);
            abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t here = s;
          const uint64_t off = stage_off;
          stage_off += (uint64_t)(SH::STAGE_BYTES >> 4);
          if (++s == STAGES) {
            s = 0;
            stage_off = 0;
            phase ^= 1;
          }
          ready = umma_bf16_x4_commit_peek(tmem_d, a_desc0 + off, b_desc0 + off, idesc, kb > 0 ? 1u : 0u, empty0 + 8 * here, full0 + 8 * s, phase);
        }
        if (ok) umma_commit(&acc_full[acc]);
        ++local;
      }
      if (!ok) {  // neither tensor memory nor the block may go before what was issued is done
        umma_commit(&drain_bar);
        mbar_wait(&drain_bar, 0);
      }
    }
  } else if (warp >= FIRST_GATHER) {
    // ---------------- rows: warp w asks for every fourth slice's
    const int w = warp - FIRST_GATHER;
    int* from = row_ids + w * NT;  // which rows of x the unit has (gathered ones)
    int next[NT / 32];             // the next unit's, asked for a unit ahead
    auto ask = [&](int unit) {
      int e = 0, r0 = 0, rows = 0;
      if (unit < n_units) group(unit, e, r0, rows);
#pragma unroll
      for (int j = 0; j < NT / 32; ++j) next[j] = lane + 32 * j < rows ? __ldcg(g.order + r0 + lane + 32 * j) : -1;
    };
    uint32_t base = 0;  // slices before this unit
    uint32_t mine = w;  // this warp's next slice
    bool ok = true;
    const bool gathered = g.order != nullptr;
    if (gathered) ask(blockIdx.x);
    for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
      int e, r0, rows;
      group(unit, e, r0, rows);
      if (rows <= 0) continue;
      const int n16 = (rows + 15) & ~15;
      if (gathered) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NT / 32; ++j) from[lane + 32 * j] = max(next[j], 0) / g.gather_div;  // (past the last: row 0, whose results are not stored)
        __syncwarp();
        ask(unit + gridDim.x);
      }
      if (lane == 0) {
        for (; mine < base + n_k; mine += GATHER_WARPS) {
          const uint32_t s = mine % STAGES;
          const int k = (int)(mine - base) * BK;
          if (mine >= STAGES && !mbar_wait_role(&empty_bar[s], (mine / STAGES - 1) & 1, ctl, 65)) {
            give_up_code(status, 65);
            abort_flag = 1;
            ok = false;
            break;
          }
          const uint32_t bar = full0 + 8 * s, dst = stage0 + A_BYTES + s * SH::STAGE_BYTES;
          if (gathered) {
            mbar_expect_tx_s(bar, n16 * BK * 2);
            for (int r = 0; r < n16; r += 4) tma_gather4_s(dst + r * BK * 2, &map_x, bar, k, *reinterpret_cast<const int4*>(from + r));
          } else {
            const int boxes = (rows + SH::BOX_ROWS - 1) / SH::BOX_ROWS;
            mbar_expect_tx_s(bar, boxes * SH::BOX_ROWS * BK * 2);
            for (int i = 0; i < boxes; ++i)
              tma_load_3d_s(dst + i * SH::BOX_ROWS * BK * 2, &map_x, bar, k, g.tiles == nullptr && g.xh != 0 ? e : 0, r0 + i * SH::BOX_ROWS);
          }
        }
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      base += n_k;
    }
    if (lane == 0) rows_asked[w] = mine;
  } else {
    // ---------------- results: warp quarter q has features 32 q .. 32 q + 31 of the tile; of its two warps one takes the pieces of
    // 32 rows with an even number, the other the odd ones
    const int q = warp & 3, half = (warp - 2) >> 2, pair = q & 1, upper = q >> 1;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
    float* traded = trade + (half * 2 + pair) * (2 * 2 * 8 * 32);
    const bool relu2 = EPI == PLAIN && g.act_limit == RL_UNARY_RELU2;
    int local = 0;
    for (int unit = blockIdx.x; unit < n_units; unit += gridDim.x) {
      int e, r0, rows;
      group(unit, e, r0, rows);
      if (rows <= 0) continue;
      const int acc = local & 1;
      // one warp polls and decides for all; the others wait at a hardware barrier, off the issue slots
      if (warp == 2) {
        const bool arrived = mbar_wait_role(&acc_full[acc], (local >> 1) & 1, ctl, 63);
        if (lane == 0) {
          if (!arrived) {
            give_up_code(status, 63);
            abort_flag = 1;
          }
          go[acc] = arrived && !*(volatile int*)&abort_flag;
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(RESULT_WARPS * 32) : "memory");
      if (!*(volatile int*)&go[acc]) break;
      tc_fence_after();
      const int n0 = (unit % blocks_n) * UNIT_N;
      const int feature = n0 + (EPI == GATED ? pair : q) * 32 + lane;
      const bool stored = feature < g.N;
      TO* to = out + (long long)(r0 + 32 * half) * g.ldo + (g.tiles == nullptr ? e * g.oh : 0) + feature;
      const bf16* gt = EPI == SIGMOID ? g.gate + (long long)(r0 + 32 * half) * g.ldg + e * g.gh + feature : nullptr;
      for (int c = 32 * half; c < rows; c += 64, to += 64 * g.ldo) {
        const int here = stored ? min(32, rows - c) : 0;  // rows of this piece that this lane stores
        bf16 factor[EPI == SIGMOID ? 32 : 1];
        if constexpr (EPI == SIGMOID) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < here) factor[j] = gt[j * g.ldg];
          gt += 64 * g.ldg;
        }
        uint32_t r[32];
        tmem_ld_32x32b_x32(lane_base + (uint32_t)(acc * NT + c), r);
        tmem_ld_wait();
        TO* p = to;
        if constexpr (EPI == GATED) {
          // of every 16 rows the first 8 are the gate's warp's to finish, the others the up's
#pragma unroll
          for (int part = 0; part < 2; ++part) {
            float* mine = traded + (part * 2 + upper) * (8 * 32) + lane, *theirs = traded + (part * 2 + (upper ^ 1)) * (8 * 32) + lane;
#pragma unroll
            for (int j = 0; j < 8; ++j) mine[j * 32] = __uint_as_float(upper ? r[16 * part + j] : r[16 * part + 8 + j]);
            // (a turn's buffer is written again after the barrier of the other turn, which both reach after reading it)
            asm volatile("bar.sync %0, 64;" ::"r"(2 + half * 2 + pair) : "memory");
            const int first = 16 * part + 8 * upper;
            p = to + first * g.ldo;
#pragma unroll
            for (int j = 0; j < 8; ++j, p += g.ldo) {
              const float own = __uint_as_float(upper ? r[16 * part + 8 + j] : r[16 * part + j]), other = theirs[j * 32];
              const float v = gated_act(upper ? other : own, upper ? own : other, g.act_alpha, g.act_limit);
              if (first + j < here) *p = from_f32<TO>(v);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j, p += g.ldo) {
            float v = __uint_as_float(r[j]);
            if constexpr (EPI == SIGMOID) v *= 1.0f / (1.0f + expf(-__bfloat162float(factor[j])));
            else if (relu2) v = unary_post(v, RL_UNARY_RELU2);
            if (j < here) *p = from_f32<TO>(v);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
      ++local;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, SH::TMEM_COLS);
  // Every role is done or has given up.  If someone gave up, the block stays until every copy that was started has landed: a stage
  // for which only one of its two halves was asked gets the other's arrival, and is waited for (bounded).
  if (threadIdx.x == 0 && *(volatile int*)&abort_flag) {
    uint32_t last = weights_asked;
    for (int w = 0; w < GATHER_WARPS; ++w) last = max(last, rows_asked[w]);
    for (uint32_t j = last > STAGES + GATHER_WARPS ? last - STAGES - GATHER_WARPS : 0; j < last; ++j) {
      const bool weights = j < weights_asked, rows = j < rows_asked[j % GATHER_WARPS];
      if (!weights && !rows) continue;
      if (!weights || !rows) mbar_arrive_s(full0 + 8 * (j % STAGES));
      mbar_wait(&full_bar[j % STAGES], (j / STAGES) & 1);
    }
  }
}

// ------------------------------------------------------------------ host side
// status: one int in device memory, 0 before the call; non-zero afterwards means a bounded wait expired (61 the copying lane,
// 62 the tensor-core issuer waiting for a stage, 63 a result warp, 64 the issuer waiting for a free accumulator, 65 a gathering
// warp) and the output is not valid.  wait_test_role, wait_test_ns: as for gemm_tc.
// [row][head][k]: boxes of 64 k x `box_rows` rows of one head (without heads: of the one there is), 128-byte swizzled.  0 on success.
static int make_rows_map(CUtensorMap* map, const Groups& g, int box_rows) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return 1;
  const int heads = g.tiles == nullptr && g.xh != 0 ? g.heads : 1;  // (without a step from head to head all read the same rows)
  cuuint64_t dims[3] = {(cuuint64_t)g.K, (cuuint64_t)heads, (cuuint64_t)g.x_rows};
  cuuint64_t strides[2] = {(cuuint64_t)(heads > 1 ? g.xh : g.ldx) * 2, (cuuint64_t)g.ldx * 2};
  cuuint32_t box[3] = {64, 1, (cuuint32_t)box_rows}, estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(g.x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : 2;
}

// Boxes of 64 k x FEATURES / 2 features of a matrix, the dimension of the smaller stride first.  0 on success.
static int make_weights_map(CUtensorMap* map, const void* w, const Always& a, int N, int K) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return 1;
  const int at_n = a.piece < a.row ? 2 : 1, at_piece = 3 - at_n;
  cuuint64_t dims[3] = {(cuuint64_t)K}, strides[2];
  cuuint32_t box[3] = {BK}, estr[3] = {1, 1, 1};
  dims[at_n] = (cuuint64_t)N, strides[at_n - 1] = (cuuint64_t)a.row * 2, box[at_n] = FEATURES / 2;
  dims[at_piece] = (cuuint64_t)a.n, strides[at_piece - 1] = (cuuint64_t)a.piece * 2, box[at_piece] = 1;
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : 2;
}

template <typename TO, int EPI, int NT, bool MORE = false>
static int launch_grouped(const void* w, const void* w2, int matrices, void* out, Groups g, const Always& always, long long max_groups, int* status,
                          int wait_test_role, unsigned int wait_test_ns, cudaStream_t stream) {
  using SH = Shape<NT>;
  WeightMaps<MORE> maps;
  CUtensorMap map_x;
  g.matrices = matrices;
  const Always dense = {nullptr, nullptr, g.K, (long long)g.N * g.K, matrices};
  maps.w2 = {};
  if (make_weights_map(&maps.w, w, dense, g.N, g.K) || (EPI == GATED && make_weights_map(&maps.w2, w2, dense, g.N, g.K)))
    RL_REFUSE(9, "grouped_gemm_tc: cannot describe the matrices to TMA");
  if (EPI != GATED) maps.w2 = maps.w;
  if constexpr (MORE) {
    // Rows of gate and up that alternate are one row of both behind each other, which one description serves (it takes the host 0.4 us); where k
    // is no multiple of a slice the first one's last slice would run into the second.
    g.piece_first = always.piece < always.row;
    const bool both = EPI == GATED && always.w2 == always.w + g.K && always.row >= 2LL * g.K && g.K % BK == 0;
    g.shift = both ? g.K : 0;
    if (make_weights_map(&maps.s, always.w, always, g.N, both ? 2 * g.K : g.K) ||
        (EPI == GATED && !both && make_weights_map(&maps.s2, always.w2, always, g.N, g.K)))
      RL_REFUSE(9, "grouped_gemm_tc: cannot describe the matrices that take every token to TMA");
    if (EPI != GATED || both) maps.s2 = maps.s;
  }
  if (g.order != nullptr ? make_matrix_map(&map_x, g.x, g.x_rows, g.K, (int)g.ldx, 1) : make_rows_map(&map_x, g, SH::BOX_ROWS))
    RL_REFUSE(9, "grouped_gemm_tc: cannot describe the rows to TMA");
  auto kern = grouped_gemm_tc_kernel<TO, EPI, NT, MORE>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::SMEM_BYTES) != cudaSuccess)
    RL_REFUSE(5, "grouped_gemm_tc: cannot get %d bytes of shared memory", SH::SMEM_BYTES);
  const int sms = rl_sm_count();
  if (sms <= 0) RL_REFUSE(10, "grouped_gemm_tc: cannot count the SMs");
  const int unit_n = EPI == GATED ? FEATURES / 2 : FEATURES;
  const long long units = max_groups * ((g.N + unit_n - 1) / unit_n);
  if (units > 0x7fffffffLL) RL_REFUSE(11, "grouped_gemm_tc: too many units of work");
  RL_LAUNCH_CHECK(rl_launch(kern, dim3((unsigned)(units < sms ? units : sms)), NUM_THREADS, SH::SMEM_BYTES, stream, maps, map_x, (TO*)out, g,
                            status, wait_test_role, (uint32_t)wait_test_ns));
  return 0;
}

static int refuse_operands(const char* what, const void* x, long long ldx, long long xh, const void* w, const void* w2, int matrices, int N, int K) {
  if (K % 8 || ldx % 8 || xh % 8) RL_REFUSE(3, "%s: k = %d or strides of %lld and %lld elements break 16-byte alignment", what, K, ldx, xh);
  if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)w2) & 15) RL_REFUSE(7, "%s: operands must be 16-byte aligned", what);
  if ((long long)matrices * N > 0x7fffffffLL) RL_REFUSE(8, "%s: %d matrices of %d rows", what, matrices, N);
  return 0;
}

// out[r] = x[order[r] / gather_div], rows of `pieces` times 16 bytes: the plan's rows next to each other, for products in which
// many feature tiles read them (a copy of four named rows takes the copy engine as long as one of 64 neighbouring ones).
__global__ void __launch_bounds__(256)
moe_gather_rows_kernel(const uint4* __restrict__ x, long long ldx, int x_rows, const int* __restrict__ order, int gather_div,
                       uint4* __restrict__ out, int n_rows, int pieces) {
  pdl_trigger();
  pdl_wait();
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < n_rows; r += gridDim.x * 8) {
    const int from = __ldcg(order + r) / gather_div;
    if (from < 0 || from >= x_rows) continue;  // (rows behind the plan's last: nobody reads them)
    const uint4* src = x + from * ldx;
    uint4* dst = out + (long long)r * pieces;
    int i = threadIdx.x & 31;
    for (; i + 96 < pieces; i += 128) {
      const uint4 a = __ldcg(src + i), b = __ldcg(src + i + 32), c = __ldcg(src + i + 64), d = __ldcg(src + i + 96);
      dst[i] = a;
      dst[i + 32] = b;
      dst[i + 64] = c;
      dst[i + 96] = d;
    }
    for (; i < pieces; i += 32) dst[i] = __ldcg(src + i);
  }
}

RL_API int rl_moe_gather_rows(const void* x, int ldx, int x_rows, const int* order, int gather_div, void* out, int n_rows, int K,
                              cudaStream_t stream) {
  if (n_rows <= 0 || K <= 0 || gather_div <= 0 || x_rows <= 0) RL_REFUSE(1, "moe_gather_rows: rows=%d of %d k=%d div=%d", n_rows, x_rows, K, gather_div);
  if (K % 8 || ldx % 8 || (((uintptr_t)x | (uintptr_t)out) & 15)) RL_REFUSE(3, "moe_gather_rows: k = %d or a row stride of %d elements breaks 16-byte alignment", K, ldx);
  const int blocks = (n_rows + 7) / 8, most = 8 * rl_sm_count();
  if (most <= 0) RL_REFUSE(10, "moe_gather_rows: cannot count the SMs");
  RL_LAUNCH_CHECK(rl_launch(moe_gather_rows_kernel, dim3(blocks < most ? blocks : most), 256, 0, stream, (const uint4*)x, (long long)ldx / 8, x_rows,
                            order, gather_div, (uint4*)out, n_rows, K / 8));
  return 0;
}

// tile_rows: the height of the plan's row tiles, 32, 128 or 256.  n_experts: matrices in w (and w2).  always: how many more the plan has, which
// take every token: feature n of the j-th at ws (ws2) + j * ws_piece + n * ws_row.
RL_API int rl_moe_gemm_tc(const void* x, int ldx, int x_rows, const int* order, int gather_div, const void* w, const void* w2, void* out, int out_dtype,
                          int ldo, const int* tiles, int max_tiles, int tile_rows, int n_experts, int N, int K, float act_alpha, float act_limit,
                          const void* ws, const void* ws2, long long ws_row, long long ws_piece, int always, int* status, int wait_test_role, unsigned int wait_test_ns, cudaStream_t stream) {
  if (max_tiles <= 0 || N <= 0 || K <= 0 || gather_div <= 0 || n_experts <= 0 || x_rows <= 0)
    RL_REFUSE(1, "moe_gemm_tc: tiles=%d experts=%d N=%d K=%d div=%d", max_tiles, n_experts, N, K, gather_div);
  if (status == nullptr || tiles == nullptr) RL_REFUSE(2, "moe_gemm_tc: no status word or no plan");
  if (int rc = refuse_operands("moe_gemm_tc", x, ldx, 0, w, w2, n_experts, N, K)) return rc;
  if (always < 0 || (always > 0 && (ws == nullptr || (ws2 == nullptr) != (w2 == nullptr) || ws_row < K || ws_piece <= 0 || ws_row % 8 || ws_piece % 8 || (((uintptr_t)ws | (uintptr_t)ws2) & 15))))
    RL_REFUSE(12, "moe_gemm_tc: %d matrices that take every token, rows %lld and pieces %lld apart", always, ws_row, ws_piece);
  const Always more = {(const bf16*)ws, (const bf16*)ws2, ws_row, ws_piece, always};
  Groups g = {};
  g.x = (const bf16*)x;
  g.ldx = ldx;
  g.x_rows = x_rows;
  g.order = order;
  g.gather_div = gather_div;
  g.tiles = tiles;
  g.ldo = ldo;
  g.N = N;
  g.K = K;
  g.act_alpha = act_alpha;
  g.act_limit = act_limit;
#define RL_GROUPED(TO, EPI, NT)                                                                                                              \
  return always > 0 ? launch_grouped<TO, EPI, NT, true>(w, w2, n_experts, out, g, more, max_tiles, status, wait_test_role, wait_test_ns, stream) \
                    : launch_grouped<TO, EPI, NT>(w, w2, n_experts, out, g, more, max_tiles, status, wait_test_role, wait_test_ns, stream)
#define RL_GROUPED_ROWS(TO, EPI)               \
  do {                                         \
    if (tile_rows == 32) RL_GROUPED(TO, EPI, 32);   \
    if (tile_rows == 128) RL_GROUPED(TO, EPI, 128); \
    if (tile_rows == 256) RL_GROUPED(TO, EPI, 256); \
    RL_REFUSE(4, "moe_gemm_tc: row tiles of %d, this kernel is built for 32, 128 and 256", tile_rows); \
  } while (0)
  if (w2 != nullptr && out_dtype == RL_BF16) RL_GROUPED_ROWS(bf16, GATED);
  if (w2 == nullptr && out_dtype == RL_F32) RL_GROUPED_ROWS(float, PLAIN);
  if (w2 == nullptr && out_dtype == RL_BF16) RL_GROUPED_ROWS(bf16, PLAIN);
#undef RL_GROUPED_ROWS
  RL_REFUSE(6, "moe_gemm_tc: unsupported output type %d (activation %d)", out_dtype, (int)(w2 != nullptr));
}

// x, out, gate: element (t, h, i) at base + t * ld + h * head stride + i.  w: [H, N, K] dense.  held: null, or for each run of seq_rows
// rows how many of them exist: only those, rounded up to 64, are computed.
RL_API int rl_head_linear_tc(const void* x, int ldx, int xh, const void* w, void* out, int ldo, int oh, const void* gate, int ldg, int gh,
                             int M, int H, int N, int K, const int* held, int seq_rows, int* status, int wait_test_role, unsigned int wait_test_ns, cudaStream_t stream) {
  if (M <= 0 || H <= 0 || N <= 0 || K <= 0) RL_REFUSE(1, "head_linear_tc: M=%d H=%d N=%d K=%d", M, H, N, K);
  if (held != nullptr && (seq_rows <= 0 || M % seq_rows)) RL_REFUSE(4, "head_linear_tc: %d rows are no runs of %d", M, seq_rows);
  if (status == nullptr) RL_REFUSE(2, "head_linear_tc: no status word");
  if (int rc = refuse_operands("head_linear_tc", x, ldx, xh, w, nullptr, H, N, K)) return rc;
  Groups g = {};
  g.x = (const bf16*)x;
  g.ldx = ldx;
  g.xh = xh;
  g.x_rows = M;
  g.gather_div = 1;
  g.heads = H;
  g.M = M;
  g.ldo = ldo;
  g.oh = oh;
  g.gate = (const bf16*)gate;
  g.ldg = ldg;
  g.gh = gh;
  g.N = N;
  g.K = K;
  g.held = held;
  g.seq_rows = seq_rows;
  const long long groups = (long long)H * (held != nullptr ? M / seq_rows * ((seq_rows + 255) / 256) : (M + 255) / 256);
  if (gate != nullptr) return launch_grouped<bf16, SIGMOID, 256>(w, nullptr, H, out, g, Always{}, groups, status, wait_test_role, wait_test_ns, stream);
  return launch_grouped<bf16, PLAIN, 256>(w, nullptr, H, out, g, Always{}, groups, status, wait_test_role, wait_test_ns, stream);
}
