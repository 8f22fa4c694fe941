// Products of 32-bit operands on the bfloat16 tensor cores (mma.sync m16n8k16), without losing digits.
//
// A float is the sum of three bfloat16 numbers exactly: the value rounded (h), what that left rounded (m), and the rest (l), 8 digits
// each.  A product of two such operands is taken as l h' + h l' + m m' + m h' + h m' + h h', smallest first; what is left out (m l' and less) is
// 2^-26 of the product, a quarter of what a float multiplication rounds away.  An operand that is bfloat16 already needs three products
// instead of six.  The tensor core cuts its sums off where an FMA rounds them, so the terms of 16 products are added up on their own and
// go into the long sum by a rounded addition (`spl_mma6_add`): against 64 bits the results are as near as a chain of FMAs.
// mma.sync does 1024 multiply-adds a cycle and SM (measured), the FMA pipe 128 with operands from registers: six products for one are
// still 1.3 times its rate, three 2.7 times, and an operand is read from shared memory once for a tile of 16 x 8 and more, where the FMA
// kernels were held up by those reads.
//
// No infinities: the difference of an infinite value and its own rounding is no number, and so is what it is multiplied into.
#pragma once
#include "common.cuh"

// Fragments of one m16n8k16 instruction in three parts.  Lane = 4 g + t holds rows g and g + 8 of A and column g of B, at four of the 16
// places of k; which number of k stands at which place is the caller's choice as long as both operands agree:
// places 0 and 1 of a lane are registers A[0]/A[1], B[0]; places 2 and 3 are A[2]/A[3], B[1].
struct SplA { uint32_t p[3][4]; };
struct SplB { uint32_t p[3][2]; };

__device__ __forceinline__ uint32_t spl_round2(float x, float y) {  // x in the lower half
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}
__device__ __forceinline__ void spl_pair(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = spl_round2(x, y);
  x -= __uint_as_float(h << 16);
  y -= __uint_as_float(h & 0xffff0000u);
  m = spl_round2(x, y);
  x -= __uint_as_float(m << 16);
  y -= __uint_as_float(m & 0xffff0000u);
  l = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);  // (at most eight digits are left: the upper half is all of it)
}
// rows g (lo) and g + 8 (hi), four numbers of k each
__device__ __forceinline__ void spl_a(SplA& a, const float (&lo)[4], const float (&hi)[4]) {
  spl_pair(lo[0], lo[1], a.p[0][0], a.p[1][0], a.p[2][0]);
  spl_pair(hi[0], hi[1], a.p[0][1], a.p[1][1], a.p[2][1]);
  spl_pair(lo[2], lo[3], a.p[0][2], a.p[1][2], a.p[2][2]);
  spl_pair(hi[2], hi[3], a.p[0][3], a.p[1][3], a.p[2][3]);
}
__device__ __forceinline__ void spl_b(SplB& b, const float (&v)[4]) {
  spl_pair(v[0], v[1], b.p[0][0], b.p[1][0], b.p[2][0]);
  spl_pair(v[2], v[3], b.p[0][1], b.p[1][1], b.p[2][1]);
}

__device__ __forceinline__ void spl_mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// d = a b + 0
__device__ __forceinline__ void spl_mma_zero(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void spl_add(float (&acc)[4], const float (&t)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] += t[i];
}

// acc[m][n] += A[m] B[n] over 16 of k, both operands in three parts.  Two chains of three instructions a tile, the small terms and the
// large: one chain of six left the tensor core waiting for its own results.
template <int M, int N>
__device__ __forceinline__ void spl_mma6_add(float (&acc)[M][N][4], const SplA (&a)[M], const SplB (&b)[N]) {
  float t[M][N][4], u[M][N][4];
#define SPL_ALL(OP, D, PA, PB)                                \
  _Pragma("unroll") for (int m = 0; m < M; ++m)               \
  _Pragma("unroll") for (int n = 0; n < N; ++n) OP(D[m][n], a[m].p[PA], b[n].p[PB])
  SPL_ALL(spl_mma_zero, t, 2, 0);
  SPL_ALL(spl_mma_zero, u, 1, 0);
  SPL_ALL(spl_mma, t, 0, 2);
  SPL_ALL(spl_mma, u, 0, 1);
  SPL_ALL(spl_mma, t, 1, 1);
  SPL_ALL(spl_mma, u, 0, 0);
#undef SPL_ALL
#pragma unroll
  for (int m = 0; m < M; ++m)
#pragma unroll
    for (int n = 0; n < N; ++n) {
      spl_add(u[m][n], t[m][n]);
      spl_add(acc[m][n], u[m][n]);
    }
}
// the same with a B that is bfloat16 (one part)
template <int N>
__device__ __forceinline__ void spl_mma3_add(float (&acc)[N][4], const SplA& a, const uint32_t (&b)[N][2]) {
  float t[N][4];
#pragma unroll
  for (int n = 0; n < N; ++n) spl_mma_zero(t[n], a.p[2], b[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) spl_mma(t[n], a.p[1], b[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) spl_mma(t[n], a.p[0], b[n]);
#pragma unroll
  for (int n = 0; n < N; ++n) spl_add(acc[n], t[n]);
}

__device__ __forceinline__ void spl_ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"((uint32_t)__cvta_generic_to_shared(smem)) : "memory");
}
__device__ __forceinline__ void spl_ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"((uint32_t)__cvta_generic_to_shared(smem)) : "memory");
}
// 16 bytes into shared memory, zeros where `here` is false
__device__ __forceinline__ void spl_cp16(void* dst, const void* src, bool here) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(here ? 16 : 0) : "memory");
}
__device__ __forceinline__ void spl_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void spl_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// ---------------------------------------------------------------- pieces that the chunked recurrences share
// Byte of number (i, j) of a [64, 64] lower triangle kept as its ten tiles of 16 x 16 bfloat16 numbers on and below the diagonal, j even (the
// one after it follows): rows of 32 bytes whose halves change places every four rows, so that eight rows' halves lie in different banks.
#define SPL_TRI_BYTES (10 * 16 * 16 * 2)
__device__ __forceinline__ int spl_tri_at(int i, int j) {
  const int tile = (i >> 4) * ((i >> 4) + 1) / 2 + (j >> 4), r = i & 15;
  return tile * 512 + r * 32 + ((((j >> 3) & 1) ^ ((r >> 2) & 1)) << 4) + (j & 7) * 2;
}
__device__ __forceinline__ void spl_tri_put(unsigned char* tri, int i, int j, float x, float y) {
  uint32_t part[3];
  spl_pair(x, y, part[0], part[1], part[2]);
#pragma unroll
  for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(tri + spl_tri_at(i, j) + e * SPL_TRI_BYTES) = part[e];
}
// tile (m, kt) as an A operand, k in order
__device__ __forceinline__ void spl_tri_a(SplA& a, const unsigned char* tri, int m, int kt, int lane) {
  const int r = lane & 15, at = (m * (m + 1) / 2 + kt) * 512 + r * 32 + (((lane >> 4) ^ ((r >> 2) & 1)) << 4);
#pragma unroll
  for (int e = 0; e < 3; ++e) spl_ldmatrix_x4(a.p[e][0], a.p[e][1], a.p[e][2], a.p[e][3], tri + e * SPL_TRI_BYTES + at);
}
// 16 rows from `rows` and 16 of k of a matrix whose parts [parts][..][ld] lie `part` elements apart, as an A operand, k in order
__device__ __forceinline__ void spl_rows_a(SplA& a, const bf16* rows, int part, int ld, int lane) {
#pragma unroll
  for (int e = 0; e < 3; ++e) spl_ldmatrix_x4(a.p[e][0], a.p[e][1], a.p[e][2], a.p[e][3], rows + e * part + (lane & 15) * ld + 8 * (lane >> 4));
}
// the same from 32-bit rows (`at`: this lane's row g and first column 2 t)
__device__ __forceinline__ void spl_rows_a(SplA& a, const float* at, int ld) {
  const float2 l0 = *reinterpret_cast<const float2*>(at), l1 = *reinterpret_cast<const float2*>(at + 8);
  const float2 h0 = *reinterpret_cast<const float2*>(at + 8 * ld), h1 = *reinterpret_cast<const float2*>(at + 8 * ld + 8);
  const float lo[4] = {l0.x, l0.y, l1.x, l1.y}, hi[4] = {h0.x, h0.y, h1.x, h1.y};
  spl_a(a, lo, hi);
}

// The end of a chunk of 64 tokens and a head of up to 128 values: warp w of eight has the sums of columns 16 w + 8 half + 2 t (and one on) of
// tokens 32 mm + 16 m + g and + 8 as acc[half][mm][m][0].  Without `w` they leave as float32 rows; with it they go through the head's
// norm and gate and leave as bfloat16, with the arithmetic of head_norm_gate in the order that it has for rows of whole fours (a lane has four
// neighbouring columns, whose squares are a chain, and the lanes' sums meet pairwise from the farthest apart): a row has the same bits
// whichever of the two makes it.  ss: 64 x 32 floats of shared memory that nobody uses any more once all threads are here.
#define RL_NOT_FUSED (-20)  // what a launcher answers, before it launches anything, where it cannot take the norm along
struct SplNorm {
  const float* w;  // [vdim]
  float eps;
  const bf16* gate;  // null, or rows gate_stride apart
  int gate_stride, act;  // 0 the gate itself, 1 the logistic function of it, 2 silu
  float scale;
};
__device__ __forceinline__ float spl_logistic(float x) { return logistic_no_branch(x); }
__device__ __forceinline__ void spl_finish(const float (&acc)[2][2][2][1][4], float* ss, int n, int t0, int h, int vdim, int col0, void* out, int out_stride,
                                           const SplNorm& norm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  if (norm.w == nullptr) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int col = col0 + 16 * warp + 8 * half + 2 * t;
      if (col >= vdim) continue;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int i = 16 * m + g;
        const float(&y)[4] = acc[half][m >> 1][m & 1][0];
        float* to = reinterpret_cast<float*>(out) + (size_t)(t0 + i) * out_stride + (size_t)h * vdim + col;
        if (i < n) *reinterpret_cast<float2*>(to) = make_float2(y[0], y[1]);
        if (i + 8 < n) *reinterpret_cast<float2*>(to + (size_t)8 * out_stride) = make_float2(y[2], y[3]);
      }
    }
    return;
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float(&y)[4] = acc[half][m >> 1][m & 1][0];
        const float first = fmaf(y[2 * e + 1], y[2 * e + 1], __fmul_rn(y[2 * e], y[2 * e]));  // the even lanes': their four's first two
        const float before = __shfl_xor_sync(0xffffffffu, first, 1);
        const float four = fmaf(y[2 * e + 1], y[2 * e + 1], fmaf(y[2 * e], y[2 * e], before));
        if (t & 1) ss[((2 * half + (t >> 1)) * 8 + warp) * 64 + 16 * m + 8 * e + g] = four;
      }
  __syncthreads();
  {
    float* at = ss + (threadIdx.x >> 6) * 8 * 64 + (threadIdx.x & 63);  // one of a row's four places in its 16 columns, of all warps
    const float s0 = at[0] + at[4 * 64], s1 = at[64] + at[5 * 64], s2 = at[2 * 64] + at[6 * 64], s3 = at[3 * 64] + at[7 * 64];
    at[0] = (s0 + s2) + (s1 + s3);
  }
  __syncthreads();
  float2 w[2];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int col = 16 * warp + 8 * half + 2 * t;
    w[half] = col < vdim ? *reinterpret_cast<const float2*>(norm.w + col) : make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = 16 * m + 8 * e + g;
      if (i >= n) continue;
      const float sum = (ss[i] + ss[16 * 64 + i]) + (ss[8 * 64 + i] + ss[24 * 64 + i]);
      const float inv = 1.0f / sqrtf(sum / (float)vdim + norm.eps);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int col = 16 * warp + 8 * half + 2 * t;
        if (col >= vdim) continue;
        const float(&y)[4] = acc[half][m >> 1][m & 1][0];
        float y0 = y[2 * e] * inv * w[half].x, y1 = y[2 * e + 1] * inv * w[half].y;
        if (norm.gate != nullptr) {
          const uint32_t raw = __ldcg(reinterpret_cast<const uint32_t*>(norm.gate + (size_t)(t0 + i) * norm.gate_stride + (size_t)h * vdim + col));
          const float g0 = __uint_as_float(raw << 16), g1 = __uint_as_float(raw & 0xffff0000u);
          y0 *= norm.act == 2 ? g0 * spl_logistic(g0) : (norm.act == 1 ? spl_logistic(g0) : g0);
          y1 *= norm.act == 2 ? g1 * spl_logistic(g1) : (norm.act == 1 ? spl_logistic(g1) : g1);
        }
        *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(out) + (size_t)(t0 + i) * out_stride + (size_t)h * vdim + col) =
            spl_round2(y0 * norm.scale, y1 * norm.scale);
      }
    }
}
