// Warp-level tensor-core pieces of the delta-rule scans (delta_rule_mma.cu, channel_delta_mma.cu): fp32 operands as sums of bf16 values, fragments,
// asynchronous copies.
//
// An fp32 value has 24 significant bits, three bf16 values have 8 each: each rounded to nearest from what the ones before it leave, the pieces add up
// to the value exactly, and a product of a piece with a bf16 number is exact in fp32.  So a product of an fp32 matrix with a bf16 one
// is three tensor-core products, one of two fp32 matrices six: a middle piece is at most 2^-9 of its value, a lowest one 2^-18, so the three pairs left
// out are within 2^-26 + 2^-36 of the product, of either sign.  (Pieces that are cut off and not rounded leave out up to 2^-21, always towards zero.)
// The lowest piece has bits to spare: the rounding errors of a value that is on its way into a product go there.
#pragma once
#include "delta_common.cuh"

namespace ats {

struct Pieces {   // of an A fragment (16 x 16): hi + mid + lo
  uint32_t hi[4], mid[4], lo[4];
};

// Two neighbouring values of a row as three words of two bf16 each; ex, ey: what their own roundings cut off.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo, float ex = 0.f, float ey = 0.f) {
  hi = pack_bf16x2(x, y);
  const float rx = x - __uint_as_float(hi << 16), ry = y - __uint_as_float(hi & 0xffff0000u);
  mid = pack_bf16x2(rx, ry);
  lo = pack_bf16x2(rx - __uint_as_float(mid << 16) + ex, ry - __uint_as_float(mid & 0xffff0000u) + ey);
}

// Accumulator tiles of columns 0..7 (a) and 8..15 (b) of a 16 x 16 block as the A operand of the next product.
__device__ __forceinline__ void split_tiles(const float (&a)[4], const float (&b)[4], Pieces& p) {
  split_pair(a[0], a[1], p.hi[0], p.mid[0], p.lo[0]);
  split_pair(a[2], a[3], p.hi[1], p.mid[1], p.lo[1]);
  split_pair(b[0], b[1], p.hi[2], p.mid[2], p.lo[2]);
  split_pair(b[2], b[3], p.hi[3], p.mid[3], p.lo[3]);
}

__device__ __forceinline__ void split_tiles(const float (&a)[4], const float (&b)[4], const float (&ea)[4], const float (&eb)[4], Pieces& p) {
  split_pair(a[0], a[1], p.hi[0], p.mid[0], p.lo[0], ea[0], ea[1]);
  split_pair(a[2], a[3], p.hi[1], p.mid[1], p.lo[1], ea[2], ea[3]);
  split_pair(b[0], b[1], p.hi[2], p.mid[2], p.lo[2], eb[0], eb[1]);
  split_pair(b[2], b[3], p.hi[3], p.mid[3], p.lo[3], eb[2], eb[3]);
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Tensor-core sums are cut off at the last place of the result: all in one direction, half a unit on average.  With c = a x b so computed, adds what was cut
// off to `small`: the same product on top of -c.  (Without it the state of a scan with fast decays is twice as far from 64 bits.)
__device__ __forceinline__ void add_rest(const float (&c)[4], float (&small)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float rest[4] = {-c[0], -c[1], -c[2], -c[3]};
  mma_bf16(rest, a, b0, b1);
#pragma unroll
  for (int e = 0; e < 4; ++e) small[e] += rest[e];
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stsm4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// 16 bytes, of which the first `bytes` are read and the rest is zero
__device__ __forceinline__ void cp_async_fill(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// A 16 x 16 fp32 matrix M in shared memory (row pitch 17) as three B operands, element [k][n] = M[n][k]; per piece a lane's 16 bytes: rows
// n = 0..7 with k = 0..7 and 8..15, then rows 8..15.
__device__ __forceinline__ void store_split_b(const float (*m)[17], int lane, uint4* dst) {
  const int g = lane >> 2, t = lane & 3;
  uint32_t hi[4], mid[4], lo[4];
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int i = g + 8 * (x >> 1), j = 2 * t + 8 * (x & 1);
    split_pair(m[i][j], m[i][j + 1], hi[x], mid[x], lo[x]);
  }
  dst[lane] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  dst[32 + lane] = make_uint4(mid[0], mid[1], mid[2], mid[3]);
  dst[64 + lane] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

// c[2] (16 rows x 16 columns) = a x b for split operands, b as store_split_b leaves it: the large products and the small ones are summed apart.
__device__ __forceinline__ void split_product(const Pieces& a, const uint4* b, int lane, float (&c)[2][4]) {
  const uint4 bh = b[lane], bm = b[32 + lane], bl = b[64 + lane];
  float small[2][4];
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[n][e] = small[n][e] = 0.f;
  mma_bf16(small[0], a.lo, bh.x, bh.y);
  mma_bf16(small[1], a.lo, bh.z, bh.w);
  mma_bf16(c[0], a.hi, bh.x, bh.y);
  mma_bf16(c[1], a.hi, bh.z, bh.w);
  mma_bf16(small[0], a.hi, bl.x, bl.y);
  mma_bf16(small[1], a.hi, bl.z, bl.w);
  mma_bf16(small[0], a.mid, bm.x, bm.y);
  mma_bf16(small[1], a.mid, bm.z, bm.w);
  mma_bf16(small[0], a.mid, bh.x, bh.y);
  mma_bf16(small[1], a.mid, bh.z, bh.w);
  mma_bf16(small[0], a.hi, bm.x, bm.y);
  mma_bf16(small[1], a.hi, bm.z, bm.w);
  add_rest(c[0], small[0], a.hi, bh.x, bh.y);
  add_rest(c[1], small[1], a.hi, bh.z, bh.w);
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[n][e] += small[n][e];
}

// u + beta x rhs, with the rounding errors of both in `err`.  beta is the diagonal of a triangular factor, and mostly its largest term by far: a tensor-core
// sum aligns its products with the largest one and loses the low bits of the others, so the product above takes the rest of the factor alone.
__device__ __forceinline__ void add_diagonal(float beta, float rhs, float& u, float& err) {
  const float p = __fmul_rn(beta, rhs), s = __fadd_rn(p, u), v = __fsub_rn(s, p);
  err = __fmaf_rn(beta, rhs, -p) + (__fsub_rn(p, __fsub_rn(s, v)) + __fsub_rn(u, v));
  u = s;
}

// Values that are not finite.  A product with a triangular factor multiplies the later tokens of its group by zeros, and zero times NaN would reach the
// earlier ones.  So once a column's U is not finite (which any value that is not finite in its right-hand side makes it), the product is taken again without
// the values from the first such token on, and what those tokens leave is NaN.  Layout of all: lane (g, t), column g or g + 8, token 8 x + 2 t + (e & 1).
__device__ __forceinline__ bool not_finite(const float (&v)[2][4]) {
  float z = 0.f;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e) z = fmaf(v[x][e], 0.f, z);
  return !(z == 0.f);
}
// Lowers `first` to the first token of each of the lane's columns that three pieces do not hold, and clears the values from there on.
__device__ __forceinline__ void clear_spoilt(float (&v)[2][4], int t, int (&first)[2]) {
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (!(fabsf(v[x][e]) < 3.38e38f)) first[e >> 1] = min(first[e >> 1], 8 * x + 2 * t + (e & 1));
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    first[c] = min(first[c], __shfl_xor_sync(0xffffffffu, first[c], 1));
    first[c] = min(first[c], __shfl_xor_sync(0xffffffffu, first[c], 2));
  }
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (8 * x + 2 * t + (e & 1) >= first[e >> 1]) v[x][e] = 0.f;
}
__device__ __forceinline__ void spoil(float (&v)[2][4], int t, const int (&first)[2]) {
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (8 * x + 2 * t + (e & 1) >= first[e >> 1]) v[x][e] = __int_as_float(0x7fffffff);
}
template <int NT>
__device__ __forceinline__ void spoil_state(float (&S)[NT][4], const int (&first)[2]) {
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (first[e >> 1] < 16) S[j][e] = __int_as_float(0x7fffffff);
}

// U [column][token] = T x (right-hand side): `t_split` the factor below its diagonal, `beta` the diagonal; eu: what the roundings of U cut off.  Returns whether
// some value of the warp is not finite; `first` then has the columns' first such tokens, from which on u is zero.
__device__ __forceinline__ bool solve_group(float (&rhs)[2][4], const uint4* t_split, const float* beta, int lane, float (&u)[2][4], float (&eu)[2][4], int (&first)[2]) {
  const int t = lane & 3;
  auto solve = [&] {
    Pieces a;
    split_tiles(rhs[0], rhs[1], a);
    split_product(a, t_split, lane, u);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const float2 be = *reinterpret_cast<const float2*>(beta + 8 * x + 2 * t);
#pragma unroll
      for (int e = 0; e < 4; ++e) add_diagonal(e & 1 ? be.y : be.x, rhs[x][e], u[x][e], eu[x][e]);
    }
  };
  solve();
  if (!__any_sync(0xffffffffu, not_finite(u))) return false;
  first[0] = first[1] = 16;
  clear_spoilt(rhs, t, first);
  solve();
  clear_spoilt(u, t, first);
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (u[x][e] == 0.f || !(fabsf(eu[x][e]) < 3.38e38f)) eu[x][e] = 0.f;
  return true;
}

}  // namespace ats
