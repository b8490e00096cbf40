// Pieces shared by the portion kernels of the delta rules (delta_rule.cu, channel_delta.cu, delta_rule_mma.cu, channel_delta_mma.cu).
#pragma once
#include "typed.cuh"

namespace ats {

constexpr int DC = 8;  // tokens per group
// Up to this many CTAs (of 64 columns) the fp32 FMA scans of 65 to 128 state rows take 32 columns a CTA instead: rows of 32 bits, bf16 heads that are no multiple of
// eight wide, and portions too short for the tensor cores (ops/delta.py).
constexpr int SCAN_FEW = 192;

// exp(rate softplus(a)), rate < 0.  The bf16 form uses the fast functions and, where exp(a) is small, the series of log(1 + x), so that a
// slow decay keeps its digits.
template <typename T>
__device__ __forceinline__ float decay_of(float a, float rate) {
  if constexpr (sizeof(T) == 4) {
    return expf(rate * (a > 20.f ? a : log1pf(expf(a))));
  } else {
    const float x = __expf(fminf(a, 20.f));
    const float l = x < 0.02f ? x * (1.f - x * (0.5f - x * (0.33333333f - 0.25f * x))) : __logf(1.f + x);
    return __expf(rate * (a > 20.f ? a : l));
  }
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }  // one packed instruction
// Keeps the compiler from requesting the shared-memory rows of more tokens than registers can hold.
__device__ __forceinline__ void pace() { asm volatile("" ::: "memory"); }

// One step of a transposing reduction over lanes: of the pair (lo, hi) this lane keeps hi when its bit `s` is set, else lo, and adds
// what the lane across sends.
__device__ __forceinline__ float keep_add(float lo, float hi, int lane, int s) {
  const bool up = (lane & s) != 0;
  return (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, s);
}

template <int BYTES> struct Bits;
template <> struct Bits<4> { using type = uint32_t; };
template <> struct Bits<8> { using type = uint2; };
template <> struct Bits<16> { using type = uint4; };

// Column c of (1 + M)^-1 for the unit lower triangular system M_ij = beta_i kk[i][j], j < i, by forward substitution.
template <typename KK>
__device__ __forceinline__ void inverse_column(const float (&beta)[DC], const KK& kk, int c, float (&y)[DC]) {
#pragma unroll
  for (int i = 0; i < DC; ++i) {
    float acc = i == c ? 1.f : 0.f;
#pragma unroll
    for (int j = i - 1; j >= 0; --j) acc -= beta[i] * kk[i][j] * y[j];
    y[i] = acc;
  }
}

// A portion of a prompt: ats_delta_scan (groups of DC tokens) and ats_delta_scan_mma (groups of 16).
struct ScanArgs {
  const void* mixed;
  long long ldm;
  const float* rlen;
  const float* gb;
  float* coef;             // [B, groups, H, .]: constants of a group and head, as the scan kernel wants them
  float* state;            // [B, H, dim, vdim]
  long long state_bs;
  void* o;                 // [B * L, H * vdim]
  long long ldo;
  int B, L, H, KH, dim, vdim, groups, fresh;
};

// The same with one decay per state row: ats_channel_delta (groups of DC tokens), ats_channel_delta_mma (groups of 16, another layout of coef).
struct ChannelArgs {
  const void* mixed;       // [B * L, ldm] convolved q, k, v
  long long ldm;
  const float* rlen;       // [B * L, 2 * KH] dim^-1/2 / |q|, 1 / |k|
  const float* gb;         // [B * L, 2 * H]: step size at H + h
  const void* a;           // [B * L, lda]: decay input of head h at h * dim
  long long lda;
  const float* neg_rate;   // [H] -exp(A)
  const float* dt_bias;    // [H * dim]
  float* coef;             // [B, groups, H, size()]
  float* state;            // [B, H, dim, vdim]
  long long state_bs;
  void* o;                 // [B * L, H * vdim]
  long long ldo;
  int B, L, H, KH, dim, vdim, groups, fresh;
  // Per group and head: [DC][2 * DC] inverse (times beta) and kq, then rows of DK floats: DC times P_i k_i, DC times P_i q_i, DC times
  // k_j g_{j+1} .. g_C, P_C; DK = 64, 128 or 256 (the state rows the scan kernel is built for), zero beyond dim.
  int DK;
  __host__ __device__ int size() const { return 2 * DC * DC + (3 * DC + 1) * DK; }
};

}  // namespace ats
