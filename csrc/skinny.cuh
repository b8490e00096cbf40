// Arguments of the decode-sized product (gemm_skinny.cu); mirrored by ops/gemm.py.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace ats {

enum SkinnyMode : int {
  kSkPart = 0,     // out [splits, T, N] fp32: the slices of the reduction
  kSkStore = 1,    // out bf16 (+ add)
  kSkF32 = 2,      // out fp32
  kSkSwiglu = 3,   // out bf16 = silu(gate) * up
  kSkSilu = 4,     // out bf16, silu on the first act_cols columns
  kSkGelu = 5,     // out bf16 = gelu_tanh(v + bias)
  kSkDyt = 6,      // x += tanh(a1 (v + bias)) w1 + b1, out bf16 = tanh(a2 x) w2 + b2
  kSkRope = 7,     // out bf16, heads of head_dim columns; those below act_cols are rotated (half-split) by the tables w1 (cosine), w2 (sine) at pos[t]
};

struct SkinnyArgs {
  int T, N, K, mode, up_offset, act_cols, head_dim;
  float alpha, a1, a2;
  int ldx;
  void* out;
  long long ldo;
  const __nv_bfloat16* add;
  long long ldadd;
  const float* bias;
  float* x;
  const float *w1, *b1, *w2, *b2;
  const int* pos;
  // RMSNorm between two products.  The first one (kSkStore) also writes next_out [T, N] = bf16(out) * next_w and, per token and tile of 128
  // columns (of 16 on the streaming kernel), the sum of squares of its bf16 results (next_parts [T, tiles]); the second one reads next_out as its activations and multiplies
  // its sums by rsqrt(sum of the scale_n parts of the token * scale_inv + scale_eps).
  const __nv_bfloat16* next_w;
  __nv_bfloat16* next_out;
  float* next_parts;
  const float* scale_parts;
  int scale_n;
  float scale_inv, scale_eps;
  int* status;
  int w_ready;   // no kernel that may still run writes w (it is no result of the same step): in a chain of launches its first tiles are requested early
};

// The product as a stream through warps (gemv_bf16.cu): out, add, scale, next and the rotation as above, next_parts per 16 columns.
int stream_product(const void* a, long long lda, const void* w, long long ldw, long long w_rows, const SkinnyArgs& p, cudaStream_t s);

}  // namespace ats
