// What the weight-streaming products of a decode step share (csrc/int4.cu, csrc/gemv_bf16.cu): a CTA owns one tile of 16 output features, or two
// that belong together, its warps split the reduction, and what a decode step does around a product is done with the sums.
#pragma once
#include "async_copy.cuh"

namespace ats {

// (weights as the 16-row operand, up to eight tokens as the columns)
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void cp_async16_or_zero(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(smem))), "l"(gmem), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(uint32_t(__cvta_generic_to_shared(smem))), "l"(gmem) : "memory");
}

// What a decode step does around its products, instead of launches of their own (all optional):
//   scale: x holds the rows of an RMSNorm before the division, x * w, and scale_parts [M, scale_n] sums of squares of x: the sums are divided by the rms;
//   next:  the RMSNorm behind the product: next_out [M, N] = (the stored values) * next_w, next_parts [M, N / 16] = their sums of squares per tile;
//   rope:  the first act_cols features are rotated in pairs half a head apart, at positions pos [M].
// With them a step of four rows has five launches a layer instead of eight (eight 2,048-wide layers with 5,632 inner columns: 298 -> 277 us).
struct StreamStep {
  const float* scale_parts;
  int scale_n;
  float scale_inv, scale_eps;
  const __nv_bfloat16* next_w;
  __nv_bfloat16* next_out;
  float* next_parts;
  const int* pos;
  const float* cos_t;
  const float* sin_t;   // [positions, head_dim / 2]
  int act_cols, head_dim;
};
enum StreamMode : int { kStreamStore = 0, kStreamSwiGLU = 1, kStreamRope = 2 };

inline bool stream_step_ok(const StreamStep& st, int mode, int N, bool add) {
  if ((st.scale_parts && st.scale_n < 1) || (st.next_out && (mode != kStreamStore || !st.next_w || !st.next_parts))) return false;
  return mode != kStreamRope || (!add && st.pos && st.cos_t && st.sin_t && st.head_dim >= 32 && (st.head_dim & 31) == 0 && N % st.head_dim == 0 && st.act_cols >= 0 &&
                                 st.act_cols % st.head_dim == 0);
}

// Tile r of this CTA: one, or with kStreamSwiGLU the gate tile and the up tile of the same features, with kStreamRope two tiles half a head apart.
template <int MODE>
__device__ __forceinline__ int stream_tile(const StreamStep& st, int N, int r) {
  const int b = int(blockIdx.x), per_half = st.head_dim >> 5;  // kStreamRope: tiles of half a head
  return MODE == kStreamRope ? b / per_half * 2 * per_half + b % per_half + r * per_half : b + r * (N >> 5);
}

// What the sums of each token are multiplied by.
template <int WARPS, int NT>
__device__ __forceinline__ void stream_scales(const StreamStep& st, int M, float* s_scale) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int m = warp; m < 8 * NT; m += WARPS) {
    float f = 1.f;
    if (st.scale_parts && m < M) {
      float ss = 0.f;
      for (int i = lane; i < st.scale_n; i += 32) ss += __ldcg(st.scale_parts + (long long)m * st.scale_n + i);
      f = rsqrtf(warp_sum(ss) * st.scale_inv + st.scale_eps);
    }
    if (lane == 0) s_scale[m] = f;
  }
}

// The sums of the warps, and what follows them, written by the whole CTA after a barrier.  STEP: with the scale and the norm behind the product; a product
// that has neither is 3 to 8 % faster without their code (4-bit 32,000 x 2,048, sixteen rows 28.7 us, with it 29.9; 1,024 x 1,024, one row 2.37 and 2.53).
template <int MODE, int WARPS, int NT, bool STEP>
__device__ __forceinline__ void stream_finish(const StreamStep& st, const float (&s_red)[WARPS][MODE == kStreamStore ? 1 : 2][8 * NT][16], const float* s_scale,
                                              const int* tile, const __nv_bfloat16* add, long long ld_add, __nv_bfloat16* out, long long ld_out, int M, int N) {
  constexpr int R = MODE == kStreamStore ? 1 : 2;
  for (int e = int(threadIdx.x); e < NT * 128; e += WARPS * 32) {  // (whole warps: 16 lanes have the tile's features of one token)
    const int m = e >> 4, f = e & 15, col = tile[0] * 16 + f;
    const bool live = m < M;
    if (!STEP && !live) continue;
    float v = 0.f, u = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      v += s_red[w][0][m][f];
      if (R == 2) u += s_red[w][R - 1][m][f];
    }
    if (STEP) {
      v *= s_scale[m];
      u *= s_scale[m];
    }
    if (MODE == kStreamRope) {
      const int half = st.head_dim >> 1, col_u = tile[R - 1] * 16 + f;
      if (!live) continue;
      if (col < st.act_cols) {
        // rounded to bf16 first: the values that a separate rotation would read
        const float a = __bfloat162float(__float2bfloat16(v)), b = __bfloat162float(__float2bfloat16(u));
        const long long at = (long long)st.pos[m] * half + col % st.head_dim;
        const float cs = st.cos_t[at], sn = st.sin_t[at];
        v = a * cs - b * sn;
        u = a * sn + b * cs;
      }
      out[(long long)m * ld_out + col] = __float2bfloat16(v);
      out[(long long)m * ld_out + col_u] = __float2bfloat16(u);
      continue;
    }
    if (MODE == kStreamSwiGLU) {
      // the gate and up products are rounded to bf16 first, as the unfused form stores them
      const float gf = __bfloat162float(__float2bfloat16(v)), uf = __bfloat162float(__float2bfloat16(u));
      v = gf / (1.f + __expf(-gf)) * uf;
    }
    if (add && live) v += __bfloat162float(add[(long long)m * ld_add + col]);
    const __nv_bfloat16 o = __float2bfloat16(v);
    if (live) out[(long long)m * ld_out + col] = o;
    if (STEP && MODE == kStreamStore && st.next_out) {
      const float b = __bfloat162float(o);
      float sq = b * b;
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
      if (live) st.next_out[(long long)m * N + col] = __float2bfloat16(b * __bfloat162float(st.next_w[col]));
      if (live && f == 0) st.next_parts[(long long)m * (N >> 4) + tile[0]] = sq;
    }
  }
}

}  // namespace ats
