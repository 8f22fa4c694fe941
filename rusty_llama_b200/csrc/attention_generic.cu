// Causal grouped-query attention over the paged cache in 32-bit arithmetic
// (src/backend/cpu.rs:363-433, src/backend/cuda.rs:157-232).
//
// It is the attention of the 32-bit path, for prompts and for decoding alike, and it
// serves any head size up to 256 in both element types.  The order of the arithmetic
// depends on nothing but the query's position and its first visible key: the visible
// keys are cut into groups of 32 counted from the first; warp w of a block takes
// groups w, w + WARPS, ... in order with an online softmax; the warps' partial results
// are then added up in warp order.  So the bits of the result do not depend on how the
// sequence was cut into steps or on what else is in the batch, nor on how many heads
// of a kv head share a block (each is computed as if alone).
//
// A block is a token and HB query heads of one kv head, so that a key or value row
// read once serves HB heads.  Bounds: a prompt, the rows' way from L2 (hence several
// heads a block); a decode step, the chain of one warp's groups (hence WARPS warps, and
// fewer heads a block until every SM has two).  32 heads of 64 on 4: prompts of 219 and
// 64 tokens 66 us a layer, a decode step of both 8.4 us and 16 from HBM (9.6 and 18 before a head
// alone read ahead; one warp per token and head, which read a key number by number: 166 us on
// average over prompts and decode steps).
//
// Cache layout of one layer: pages[page][kv_head][slot_in_page][hd]; the page of
// position p of batch sequence s is block_table[s][p / page_size].
#include "common.cuh"

RL_DEFINE_ERROR_TEXT()

#define WARPS 8  // part of the summation order

// DPL: value dimensions per lane (head sizes up to 32 DPL); HB: query heads per block; by4: the keys' rows can be read four numbers at a time;
// ALONE: see rl_attn_generic
template <typename T, int DPL, int HB, bool ALONE>
__global__ void __launch_bounds__(WARPS * 32)
attn_generic_kernel(const T* __restrict__ q, int q_stride, const T* __restrict__ k_pages,
                    const T* __restrict__ v_pages, const int* __restrict__ block_table, int table_width,
                    const int* __restrict__ tok_seq, const int* __restrict__ tok_pos, T* __restrict__ out, int out_stride,
                    int H, int K, int hd, int page_size, int window, float scale, bool by4) {
  static_assert(!ALONE || HB == 1, "a head alone");
  constexpr int AHEAD = 32 / DPL;  // rows of values that a lane asks for at a time
  extern __shared__ __align__(16) float sm[];
  const int hd4 = (hd + 3) & ~3;
  float* q_s = sm;                              // [HB][hd4]
  float* p_s = q_s + HB * hd4;                  // [WARPS][HB][32]
  float* acc_s = p_s + WARPS * HB * 32;         // [WARPS][HB][hd]
  float* ml_s = acc_s + WARPS * HB * hd;        // [WARPS][HB][2]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = H / K, blocks_per_kv = (G + HB - 1) / HB;
  const int t = blockIdx.x, kh = blockIdx.y / blocks_per_kv;
  const int g0 = (blockIdx.y - kh * blocks_per_kv) * HB;
  const int n_heads = min(HB, G - g0), h0 = kh * G + g0;
  const int pos = tok_pos[t];
  const int* table = block_table + (size_t)tok_seq[t] * table_width;
  for (int i = threadIdx.x; i < HB * hd4; i += WARPS * 32) {
    const int h = i / hd4, d = i - h * hd4;
    q_s[i] = (h < n_heads && d < hd) ? to_f32(q[(size_t)t * q_stride + (size_t)(h0 + h) * hd + d]) : 0.f;
  }
  __syncthreads();

  // keep when pos - key < window (src/backend/cpu.rs:404-409)
  const int first = (window != 0 && pos + 1 > window) ? pos + 1 - window : 0;
  float m[HB], l[HB], acc[HB][DPL];
#pragma unroll
  for (int h = 0; h < HB; ++h) {
    m[h] = -INFINITY;
    l[h] = 0.f;
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[h][i] = 0.f;
  }
  float* ps = p_s + warp * HB * 32;

  for (int base = first + 32 * warp; base <= pos; base += 32 * WARPS) {
    const int key = base + lane;
    const bool valid = key <= pos;
    float s[HB];
#pragma unroll
    for (int h = 0; h < HB; ++h) s[h] = 0.f;
    const size_t row = valid ? (((size_t)table[key / page_size] * K + kh) * page_size + key % page_size) * hd : 0;
    if (valid) {
      const T* kr = k_pages + row;
      if (ALONE && by4) {  // sixteen pieces of the row on their way at a time
        for (int i0 = 0; i0 < hd; i0 += 64) {
          float kv[16][4];
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (i0 + 4 * j < hd) load4(kr + i0 + 4 * j, kv[j]);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (i0 + 4 * j >= hd) break;
            const float4 qv = *reinterpret_cast<const float4*>(q_s + i0 + 4 * j);
            s[0] = fmaf(qv.x, kv[j][0], s[0]);
            s[0] = fmaf(qv.y, kv[j][1], s[0]);
            s[0] = fmaf(qv.z, kv[j][2], s[0]);
            s[0] = fmaf(qv.w, kv[j][3], s[0]);
          }
        }
      } else if (by4) {
#pragma unroll 4
        for (int i = 0; i < hd; i += 4) {
          float kv[4];
          load4(kr + i, kv);
#pragma unroll
          for (int h = 0; h < HB; ++h) {
            const float4 qv = *reinterpret_cast<const float4*>(q_s + h * hd4 + i);
            s[h] = fmaf(qv.x, kv[0], s[h]);
            s[h] = fmaf(qv.y, kv[1], s[h]);
            s[h] = fmaf(qv.z, kv[2], s[h]);
            s[h] = fmaf(qv.w, kv[3], s[h]);
          }
        }
      } else {
        for (int i = 0; i < hd; ++i) {
          const float kv = to_f32(kr[i]);
#pragma unroll
          for (int h = 0; h < HB; ++h) s[h] = fmaf(q_s[h * hd4 + i], kv, s[h]);
        }
      }
    }
    // a head alone: the values' rows do not wait for the probabilities, nor a row's place for the table (the lane that has its key knows it)
    const int count = min(32, pos - base + 1);
    float ahead[ALONE ? AHEAD : 1][DPL];
    auto ask = [&](int j0) {
#pragma unroll
      for (int j = 0; j < AHEAD; ++j) {
        const T* vr = v_pages + __shfl_sync(0xffffffffu, (unsigned long long)row, j0 + j);
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
          const int dim = lane + 32 * i;
          ahead[ALONE ? j : 0][i] = (dim < hd && j0 + j < count) ? to_f32(vr[dim]) : 0.f;
        }
      }
    };
    if constexpr (ALONE) ask(0);
#pragma unroll
    for (int h = 0; h < HB; ++h) {
      const float v = valid ? __fmul_rn(s[h], scale) : -INFINITY;  // (rounded here in every form of this kernel, not inside a later sum)
      const float m_new = fmaxf(m[h], warp_max(v));  // finite: the group holds at least key `base`
      const float alpha = expf(m[h] - m_new);        // 0 for the first group, where m is -inf
      const float p = valid ? expf(v - m_new) : 0.f;
      l[h] = fmaf(l[h], alpha, warp_sum(p));
      m[h] = m_new;
      ps[h * 32 + lane] = p;
#pragma unroll
      for (int i = 0; i < DPL; ++i) acc[h][i] *= alpha;
    }
    __syncwarp();
    if constexpr (ALONE) {
      for (int j0 = 0; j0 < count; j0 += AHEAD) {
        if (j0) ask(j0);
#pragma unroll
        for (int j = 0; j < AHEAD; j += 4) {
          if (j0 + j >= count) break;
          const float4 p = *reinterpret_cast<const float4*>(ps + j0 + j);
#pragma unroll
          for (int i = 0; i < DPL; ++i) {
            acc[0][i] = fmaf(p.x, ahead[ALONE ? j : 0][i], acc[0][i]);
            acc[0][i] = fmaf(p.y, ahead[ALONE ? j + 1 : 0][i], acc[0][i]);
            acc[0][i] = fmaf(p.z, ahead[ALONE ? j + 2 : 0][i], acc[0][i]);
            acc[0][i] = fmaf(p.w, ahead[ALONE ? j + 3 : 0][i], acc[0][i]);
          }
        }
      }
      __syncwarp();
      continue;
    }
#pragma unroll 2
    for (int j0 = 0; j0 < count; j0 += 4) {
      float v[4][DPL];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kj = min(base + j0 + j, pos);  // (past the last key: nothing is read, the probability is zero)
        const T* vr = v_pages + (((size_t)table[kj / page_size] * K + kh) * page_size + kj % page_size) * hd;
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
          const int dim = lane + 32 * i;
          v[j][i] = (dim < hd && j0 + j < count) ? to_f32(vr[dim]) : 0.f;
        }
      }
#pragma unroll
      for (int h = 0; h < HB; ++h) {
        const float4 p = *reinterpret_cast<const float4*>(ps + h * 32 + j0);
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
          acc[h][i] = fmaf(p.x, v[0][i], acc[h][i]);
          acc[h][i] = fmaf(p.y, v[1][i], acc[h][i]);
          acc[h][i] = fmaf(p.z, v[2][i], acc[h][i]);
          acc[h][i] = fmaf(p.w, v[3][i], acc[h][i]);
        }
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int h = 0; h < HB; ++h) {
    if (lane == 0) {
      ml_s[(warp * HB + h) * 2] = m[h];  // -inf: the warp had no group
      ml_s[(warp * HB + h) * 2 + 1] = l[h];
    }
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      const int dim = lane + 32 * i;
      if (dim < hd) acc_s[(warp * HB + h) * hd + dim] = acc[h][i];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n_heads * hd; i += WARPS * 32) {
    const int h = i / hd, d = i - h * hd;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) M = fmaxf(M, ml_s[(w * HB + h) * 2]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float f = expf(ml_s[(w * HB + h) * 2] - M);  // 0 for a warp without a group
      den = fmaf(f, ml_s[(w * HB + h) * 2 + 1], den);
      num = fmaf(f, acc_s[(w * HB + h) * hd + d], num);
    }
    out[(size_t)t * out_stride + (size_t)(h0 + h) * hd + d] = from_f32<T>(num / den);
  }
}

template <typename T, int DPL, int HB, bool ALONE = false>
static int launch_attn_generic(const void* q, int q_stride, const void* k_pages, const void* v_pages, const int* block_table,
                               int table_width, const int* tok_seq, const int* tok_pos, void* out, int out_stride, int n_tokens,
                               int H, int K, int hd, int page_size, int window, float scale, cudaStream_t stream) {
  const int G = H / K, gy = K * ((G + HB - 1) / HB);
  if (gy > 65535) RL_REFUSE(4, "attn_generic: %d heads exceed the grid", H);
  const size_t smem = (size_t)(HB * ((hd + 3) & ~3) + WARPS * HB * (32 + hd + 2)) * sizeof(float);
  auto kern = attn_generic_kernel<T, DPL, HB, ALONE>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    RL_REFUSE(7, "attn_generic: cannot get %zu bytes of shared memory", smem);
  const bool by4 = hd % 4 == 0 && (uintptr_t)k_pages % (4 * sizeof(T)) == 0;
  kern<<<dim3(n_tokens, gy), WARPS * 32, smem, stream>>>((const T*)q, q_stride, (const T*)k_pages, (const T*)v_pages, block_table,
                                                         table_width, tok_seq, tok_pos, (T*)out, out_stride, H, K, hd, page_size,
                                                         window, scale, by4);
  RL_LAUNCH_RESULT();
}

RL_API int rl_attn_generic(const void* q, int dtype, int q_stride, const void* k_pages, const void* v_pages,
                           const int* block_table, int table_width, const int* tok_seq, const int* tok_pos,
                           void* out, int out_stride, int n_tokens, int H, int K, int hd, int page_size,
                           int window, float scale, int sms, cudaStream_t stream) {
  if (n_tokens <= 0 || H <= 0 || K <= 0 || hd <= 0 || page_size <= 0 || sms <= 0)
    RL_REFUSE(1, "attn_generic: T=%d H=%d K=%d hd=%d page=%d on %d SMs", n_tokens, H, K, hd, page_size, sms);
  if (H % K) RL_REFUSE(2, "attn_generic: %d query heads are not a multiple of %d kv heads", H, K);
  if (hd > 256) RL_REFUSE(3, "attn_generic: head size %d exceeds 256", hd);
  if (H > 65535) RL_REFUSE(4, "attn_generic: %d heads exceed 65535", H);
  if (window < 0) RL_REFUSE(5, "attn_generic: negative window");
  if (dtype != RL_BF16 && dtype != RL_F32) RL_REFUSE(6, "attn_generic: unknown dtype %d", dtype);
  // heads a block: as many as the registers hold (16 sums a lane) while every SM has two blocks
  const int dpl = hd <= 64 ? 2 : hd <= 128 ? 4 : 8, G = H / K;
  int hb = 16 / dpl;
  while (hb > 1 && (hb / 2 >= G || (long long)n_tokens * K * ((G + hb - 1) / hb) < 2LL * sms)) hb /= 2;
  // A head alone and no more blocks than the SMs hold at once (two each, at 128 registers a thread): all of a key's pieces and the values' rows are
  // asked for ahead.  One token in 32 heads of 64 over 2000 keys 58 and 44 us, eight over 300 19.7 and 15.2; 384 blocks over 300 keys 24 and 26,
  // 1600 94 and 126, where the registers cost more blocks at a time than the waits.  (Of larger heads none gained: 40 of 128 over 300 keys 19.5 both.)
  if (dpl == 2 && hb == 1 && (long long)n_tokens * H <= 2LL * sms)
    return dtype == RL_BF16 ? launch_attn_generic<bf16, 2, 1, true>(q, q_stride, k_pages, v_pages, block_table, table_width, tok_seq, tok_pos, out, out_stride,
                                                                    n_tokens, H, K, hd, page_size, window, scale, stream)
                            : launch_attn_generic<float, 2, 1, true>(q, q_stride, k_pages, v_pages, block_table, table_width, tok_seq, tok_pos, out, out_stride,
                                                                     n_tokens, H, K, hd, page_size, window, scale, stream);
#define RL_GENERIC(D, B)                                                                                                              \
  if (dpl == D && hb == B)                                                                                                            \
    return dtype == RL_BF16 ? launch_attn_generic<bf16, D, B>(q, q_stride, k_pages, v_pages, block_table, table_width, tok_seq, tok_pos, \
                                                              out, out_stride, n_tokens, H, K, hd, page_size, window, scale, stream)   \
                            : launch_attn_generic<float, D, B>(q, q_stride, k_pages, v_pages, block_table, table_width, tok_seq, tok_pos, \
                                                               out, out_stride, n_tokens, H, K, hd, page_size, window, scale, stream)
  RL_GENERIC(2, 8);
  RL_GENERIC(2, 4);
  RL_GENERIC(2, 2);
  RL_GENERIC(2, 1);
  RL_GENERIC(4, 4);
  RL_GENERIC(4, 2);
  RL_GENERIC(4, 1);
  RL_GENERIC(8, 2);
  RL_GENERIC(8, 1);
#undef RL_GENERIC
  RL_REFUSE(8, "attn_generic: no kernel for %d heads of %d", hb, hd);
}
