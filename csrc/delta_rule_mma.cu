// Gated delta rule (delta_rule.cu has the recurrence): portions of a prompt on the tensor cores, bf16 rows of up to 128 state rows
//
// With S the state before a group of DM = 16 tokens, G_i = g_1 .. g_i, D_ij = g_{j+1} .. g_i,
//
//   U = T (V - diag(G / |k|) K S),   O = diag(G c / |q|) Q S + R U,   S <- G_C S + K^T diag(D_C / |k|) U
//
// T = (1 + tril(beta D K K^T))^-1 beta and R = tril(D Q K^T) do not depend on the value column; delta_pairs_mma computes them for all groups at
// once.  What is left is a chain of groups, each three products with the state.
//
// The state stays in registers as the accumulator tiles of S^T: a warp owns 16 value columns (the 16 rows of its tiles), all state rows and so the
// whole chain of its columns; no warp waits for another but for the rows that they share.  An accumulator tile of m16n8k16 has the
// layout of half an A operand, so S^T multiplies K^T and Q^T (k, q rows by ldmatrix), the right-hand side T^T and U^T R^T and K without leaving the
// registers.  k and q are bf16 as they come; S, the right-hand side, U, T and R are fp32 and enter as exact sums of three bf16 pieces (delta_mma.cuh),
// products of the leading pieces and of the others summed apart; the diagonal of T and the state's decay are fp32 FMAs, since tensor-core sums are cut off,
// not rounded, and the rounding errors of U and of U D / |k| go into the state with them.
//
// What bounds it is the warp-level MMA pipe (some 13 cycles an instruction and SM quarter; 200 a group and warp) and, with one warp a quarter, the chain of
// dependent products.  Scan and pairs, us, fp32 FMA form (delta_rule.cu) / this one, 128 x 128 states: 8 sequences of 2,048 tokens, 16 heads 1,129 / 454, 12 of
// 1,000 878 / 357, 3 of 1,501 449 / 204, one of 2,048 435 / 268, one of 512, 8 heads 116 / 77, one of 64 24 / 22.  State against 64 bits: 0.65 to 0.86 of the FMA form's
// error on average, from slow decays to those that forget a token at once; read-outs 1.66e-3 (their rounding to bf16) on both.
#include "delta_mma.cuh"

namespace ats {

namespace {

constexpr int DM = 16;                          // tokens per group
constexpr int DM_B = 3 * 32 * 16;               // bytes of a 16 x 16 matrix as split B operand
constexpr int DM_VEC = 4 * DM + 4;              // floats: G_i / |k_i|, G_i c / |q_i|, D_Ci / |k_i|, the diagonal of T (the step sizes), then G_C
constexpr int DM_COEF = 2 * DM_B + DM_VEC * 4;  // bytes per group and head: T without its diagonal, R, the vectors
constexpr int DM_COLS = 64;                     // value columns of a CTA
constexpr int DM_STAGES = 3;

// One warp per (group, kv head, sequence): 16 x 16 products of the keys with keys and queries, then per value head T and R.
__global__ void __launch_bounds__(128) delta_pairs_mma_kernel(const ScanArgs p) {
  pdl_prologue();
  __shared__ float s_kk[4][DM][17], s_kq[4][DM][17];
  __shared__ float s_m[4][2][2][DM][17];   // [warp][head of the pair][T, R]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rep = p.H / p.KH;
  const long long w = blockIdx.x * 4ll + warp;
  if (w >= (long long)p.B * p.groups * p.KH) return;   // whole warp; only __syncwarp below
  const int kh = int(w % p.KH), grp = int((w / p.KH) % p.groups), b = int(w / p.KH / p.groups);
  const int t0 = grp * DM, n = min(DM, p.L - t0);
  const long long row0 = (long long)b * p.L + t0;
  const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(p.mixed) + row0 * p.ldm + (long long)kh * p.dim;
  const __nv_bfloat16* k = q + (long long)p.KH * p.dim;
  const float* rl = p.rlen + row0 * 2 * p.KH;
  const int g = lane >> 2, t = lane & 3;
  {
    // The order of the reduction is permuted so that a lane's 16-byte piece of a row serves two steps, as A and as B operand.
    float kk[2][4] = {}, kq[2][4] = {};
    for (int d = 8 * t; d < ((p.dim + 31) & ~31); d += 32) {
      uint4 k0 = make_uint4(0, 0, 0, 0), k1 = k0, q0 = k0, q1 = k0;
      if (d < p.dim) {
        if (g < n) k0 = *reinterpret_cast<const uint4*>(k + g * p.ldm + d), q0 = *reinterpret_cast<const uint4*>(q + g * p.ldm + d);
        if (g + 8 < n) k1 = *reinterpret_cast<const uint4*>(k + (g + 8) * p.ldm + d), q1 = *reinterpret_cast<const uint4*>(q + (g + 8) * p.ldm + d);
      }
      const uint32_t ka[2][4] = {{k0.x, k1.x, k0.y, k1.y}, {k0.z, k1.z, k0.w, k1.w}}, qa[2][4] = {{q0.x, q1.x, q0.y, q1.y}, {q0.z, q1.z, q0.w, q1.w}};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        mma_bf16(kk[0], ka[s], ka[s][0], ka[s][2]);
        mma_bf16(kk[1], ka[s], ka[s][1], ka[s][3]);
        mma_bf16(kq[0], qa[s], ka[s][0], ka[s][2]);
        mma_bf16(kq[1], qa[s], ka[s][1], ka[s][3]);
      }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = g + 8 * (e >> 1), j = 8 * x + 2 * t + (e & 1);
        const float rkj = j < n ? rl[(long long)j * 2 * p.KH + p.KH + kh] : 0.f;
        const float rki = i < n ? rl[(long long)i * 2 * p.KH + p.KH + kh] : 0.f, rqi = i < n ? rl[(long long)i * 2 * p.KH + kh] : 0.f;
        s_kk[warp][i][j] = kk[x][e] * rki * rkj;
        s_kq[warp][i][j] = kq[x][e] * rqi * rkj;
      }
  }
  __syncwarp();
  // lane = (value head of a pair, column c)
  const int c = lane & 15, r = lane >> 4;
  const float rk = c < n ? rl[(long long)c * 2 * p.KH + p.KH + kh] : 0.f, rq = c < n ? rl[(long long)c * 2 * p.KH + kh] : 0.f;
  for (int r0 = 0; r0 < rep; r0 += 2) {
    const int h = kh * rep + min(r0 + r, rep - 1);
    uint8_t* co = reinterpret_cast<uint8_t*>(p.coef) + (((long long)b * p.groups + grp) * p.H + kh * rep + r0) * DM_COEF;
    float gd[DM], beta[DM], y[DM], bc = 0.f;
#pragma unroll
    for (int i = 0; i < DM; ++i) {
      gd[i] = i < n ? p.gb[(row0 + i) * 2 * p.H + h] : 1.f;
      beta[i] = i < n ? p.gb[(row0 + i) * 2 * p.H + p.H + h] : 0.f;
      if (i == c) bc = beta[i];
    }
    // column c of (1 + M)^-1, M_ij = beta_i D_ij kk_ij, by forward substitution; times beta_c
#pragma unroll
    for (int i = 0; i < DM; ++i) {
      float acc = i == c ? 1.f : 0.f, dec = 1.f;
#pragma unroll
      for (int j = i - 1; j >= 0; --j) {
        dec *= gd[j + 1];
        acc -= beta[i] * dec * s_kk[warp][i][j] * y[j];
      }
      y[i] = acc;
      s_m[warp][r][0][i][c] = i <= c ? 0.f : acc * bc;
    }
    float dec = 1.f, G = 1.f, GC = 1.f;
#pragma unroll
    for (int i = 0; i < DM; ++i) {
      if (i > c) dec *= gd[i];
      s_m[warp][r][1][i][c] = i >= c ? dec * s_kq[warp][i][c] : 0.f;
      if (i <= c) G *= gd[i];
      GC *= gd[i];
    }
    if (r0 + r < rep) {
      float* vec = reinterpret_cast<float*>(co + r * DM_COEF + 2 * DM_B);
      vec[c] = G * rk;
      vec[DM + c] = G * rq;
      vec[2 * DM + c] = dec * rk;   // dec has become g_{c+1} .. g_C
      vec[3 * DM + c] = bc;
      if (c == 0) vec[4 * DM] = GC;
    }
    __syncwarp();
    for (int x = 0; x < 2 && r0 + x < rep; ++x)
#pragma unroll
      for (int m = 0; m < 2; ++m) store_split_b(s_m[warp][x][m], lane, reinterpret_cast<uint4*>(co + x * DM_COEF + m * DM_B));
    __syncwarp();
  }
}

// DK: state rows of the tiles (dim rounded up to 64 or 128).
template <int DK>
__global__ void __launch_bounds__(128, 2) delta_scan_mma_kernel(const ScanArgs p) {
  pdl_prologue();
  constexpr int NT = DK / 8, KS = DK / 16, PITCH = DK * 2 + 16, VPITCH = DM_COLS * 2 + 16;   // (odd numbers of 16-byte pieces: no bank conflicts)
  constexpr int K_AT = 0, Q_AT = DM * PITCH, V_AT = 2 * DM * PITCH, C_AT = V_AT + DM * VPITCH, STAGE = C_AT + DM_COEF;
  constexpr int OPITCH = 48;
  __shared__ __align__(16) uint8_t s_ring[DM_STAGES][STAGE];
  __shared__ __align__(16) uint8_t s_out[4][DM * OPITCH];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int h = blockIdx.y, b = blockIdx.z, kh = h / (p.H / p.KH);
  const int cta0 = blockIdx.x * DM_COLS, col0 = cta0 + warp * 16;
  float S[NT][4];   // tile j: rows = columns col0 + g (+ 8) of the state, columns = its rows 8 j + 2 t, + 1
  float* st = p.state + (long long)b * p.state_bs + (long long)h * p.dim * p.vdim;
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * j + 2 * t + (e & 1), col = col0 + g + 8 * (e >> 1);
      S[j][e] = !p.fresh && d < p.dim && col < p.vdim ? st[(long long)d * p.vdim + col] : 0.f;
    }
  const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(p.mixed) + (long long)b * p.L * p.ldm;
  const uint8_t* cbase = reinterpret_cast<const uint8_t*>(p.coef) + ((long long)b * p.groups * p.H + h) * DM_COEF;
  auto request = [&](int grp) {
    if (grp < p.groups) {
      const uint32_t at = smem_u32(s_ring[grp % DM_STAGES]);
      const int t0 = grp * DM, n = min(DM, p.L - t0);
#pragma unroll
      for (int i = tid; i < 2 * DM * (DK / 8); i += 128) {
        const int which = i / (DM * (DK / 8)), tok = i / (DK / 8) % DM, d = i % (DK / 8) * 8;
        const bool in = tok < n && d < p.dim;
        cp_async_fill(at + (which ? Q_AT : K_AT) + tok * PITCH + d * 2,
                      in ? base + (long long)(t0 + tok) * p.ldm + (long long)(which ? kh : p.KH + kh) * p.dim + d : base, in ? 16 : 0);
      }
      {
        const int tok = tid >> 3, c = (tid & 7) * 8;
        const bool in = tok < n && cta0 + c < p.vdim;
        cp_async_fill(at + V_AT + tok * VPITCH + c * 2, in ? base + (long long)(t0 + tok) * p.ldm + 2 * p.KH * p.dim + (long long)h * p.vdim + cta0 + c : base, in ? 16 : 0);
      }
      const uint8_t* src = cbase + (long long)grp * p.H * DM_COEF;
      for (int i = tid; i < DM_COEF / 16; i += 128) cp_async_fill(at + C_AT + i * 16, src + i * 16, 16);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");   // (empty behind the last group: the count of groups in flight stays the same)
  };
#pragma unroll
  for (int i = 0; i < DM_STAGES - 1; ++i) request(i);
  // ldmatrix: lane l points at row l % 8 of block l / 8.  Blocks of a 16 x 16 piece of rows: as B operand [state row][token] tokens 0..7 and 8..15 outer,
  // state rows inner; transposed ([token][state row], and the values) tokens inner.
  const uint32_t plain = uint32_t(((lane & 7) + (lane >> 4) * 8) * PITCH + (lane >> 3 & 1) * 16);
  const uint32_t turned = uint32_t(((lane & 7) + (lane >> 3 & 1) * 8) * PITCH + (lane >> 4) * 16);
  const uint32_t vturned = uint32_t(((lane & 7) + (lane >> 3 & 1) * 8) * VPITCH + (lane >> 4) * 16 + warp * 32);
  const uint32_t out_at = smem_u32(s_out[warp]);
  for (int grp = 0; grp < p.groups; ++grp) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DM_STAGES - 2) : "memory");
    __syncthreads();   // this group's rows are there for everyone, and everyone is done with the group before
    request(grp + DM_STAGES - 1);
    const uint8_t* stage = s_ring[grp % DM_STAGES];
    const uint32_t at = smem_u32(stage);
    const uint4* mt = reinterpret_cast<const uint4*>(stage + C_AT);
    const uint4* mr = reinterpret_cast<const uint4*>(stage + C_AT + DM_B);
    const float* vec = reinterpret_cast<const float*>(stage + C_AT + 2 * DM_B);
    const int t0 = grp * DM, n = min(DM, p.L - t0);
    // S^T K^T and S^T Q^T: [column][token]; the leading pieces apart from the others
    float sk[2][4] = {}, sq[2][4] = {}, ek[2][4] = {}, eq[2][4] = {};
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      Pieces a;
      uint32_t kb[4], qb[4];
      split_tiles(S[2 * s], S[2 * s + 1], a);
      ldsm4(kb, at + K_AT + plain + s * 32);
      ldsm4(qb, at + Q_AT + plain + s * 32);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mma_bf16(sk[x], a.hi, kb[2 * x], kb[2 * x + 1]);
        mma_bf16(sq[x], a.hi, qb[2 * x], qb[2 * x + 1]);
        mma_bf16(ek[x], a.lo, kb[2 * x], kb[2 * x + 1]);
        mma_bf16(eq[x], a.lo, qb[2 * x], qb[2 * x + 1]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mma_bf16(ek[x], a.mid, kb[2 * x], kb[2 * x + 1]);
        mma_bf16(eq[x], a.mid, qb[2 * x], qb[2 * x + 1]);
      }
    }
    float u[2][4], eu[2][4];
    int first[2];
    bool spoilt;
    Pieces a;
    {
      uint32_t vv[4];   // tokens 0..7 / 8..15 of column g, then of column g + 8
      ldsm4_t(vv, at + V_AT + vturned);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 gk = *reinterpret_cast<const float2*>(vec + 8 * x + 2 * t), lo = unpack_bf16x2(vv[x]), hi = unpack_bf16x2(vv[2 + x]);
        sk[x][0] = lo.x - gk.x * (sk[x][0] + ek[x][0]);
        sk[x][1] = lo.y - gk.y * (sk[x][1] + ek[x][1]);
        sk[x][2] = hi.x - gk.x * (sk[x][2] + ek[x][2]);
        sk[x][3] = hi.y - gk.y * (sk[x][3] + ek[x][3]);
      }
      spoilt = solve_group(sk, mt, vec + 3 * DM, lane, u, eu, first);
    }
    {   // the state first: the next group waits for it
      float w[2][4], ew[2][4];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 dk = *reinterpret_cast<const float2*>(vec + 2 * DM + 8 * x + 2 * t);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float f = e & 1 ? dk.y : dk.x;
          w[x][e] = u[x][e] * f;
          ew[x][e] = fmaf(u[x][e], f, -w[x][e]) + eu[x][e] * f;
        }
      }
      split_tiles(w[0], w[1], ew[0], ew[1], a);
      const float GC = vec[4 * DM];
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        uint32_t kt[4];
        ldsm4_t(kt, at + K_AT + turned + s * 32);
        float d[2][4] = {}, f[2][4] = {};
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          mma_bf16(d[x], a.hi, kt[2 * x], kt[2 * x + 1]);
          mma_bf16(f[x], a.lo, kt[2 * x], kt[2 * x + 1]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          mma_bf16(f[x], a.mid, kt[2 * x], kt[2 * x + 1]);
          add_rest(d[x], f[x], a.hi, kt[2 * x], kt[2 * x + 1]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[2 * s + x][e] = fmaf(S[2 * s + x][e], GC, f[x][e]) + d[x][e];
      }
    }
    {
      float o[2][4];
      split_tiles(u[0], u[1], a);
      split_product(a, mr, lane, o);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 gq = *reinterpret_cast<const float2*>(vec + DM + 8 * x + 2 * t);
        o[x][0] += gq.x * (sq[x][0] + eq[x][0]);
        o[x][1] += gq.y * (sq[x][1] + eq[x][1]);
        o[x][2] += gq.x * (sq[x][2] + eq[x][2]);
        o[x][3] += gq.y * (sq[x][3] + eq[x][3]);
      }
      if (spoilt) {
        spoil(o, t, first);
        spoil_state(S, first);
      }
      // [token][column] in shared memory: blocks (tokens 0..7, columns 0..7), (0..7, 8..15), (8..15, 0..7), (8..15, 8..15)
      stsm4_t(out_at + ((lane & 7) + (lane >> 4) * 8) * OPITCH + (lane >> 3 & 1) * 16, pack_bf16x2(o[0][0], o[0][1]), pack_bf16x2(o[0][2], o[0][3]),
              pack_bf16x2(o[1][0], o[1][1]), pack_bf16x2(o[1][2], o[1][3]));
      __syncwarp();
      const int tok = lane >> 1, col = col0 + (lane & 1) * 8;
      const uint4 v = *reinterpret_cast<const uint4*>(s_out[warp] + tok * OPITCH + (lane & 1) * 16);
      if (tok < n && col < p.vdim)
        *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.o) + ((long long)b * p.L + t0 + tok) * p.ldo + (long long)h * p.vdim + col) = v;
      __syncwarp();
    }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * j + 2 * t + (e & 1), col = col0 + g + 8 * (e >> 1);
      if (d < p.dim && col < p.vdim) st[(long long)d * p.vdim + col] = S[j][e];
    }
}

}  // namespace
}  // namespace ats

using namespace ats;

// bf16 rows whose parts are whole 16-byte pieces (dim, vdim, ldm, ldo multiples of 8, mixed and o 16-byte aligned), dim up to 128, p->groups groups of 16
// tokens; coef: 836 floats per (sequence, group, head), 16-byte aligned.
ATS_API int ats_delta_scan_mma(const ScanArgs* p, int fp32, void* stream) {
  if (p->B <= 0 || p->L <= 0) return 0;
  if (fp32 || p->groups != (p->L + DM - 1) / DM || p->KH < 1 || p->H % p->KH || p->dim < 1 || p->dim > 128 || ((p->dim | p->vdim | p->ldm | p->ldo) & 7) ||
      ((reinterpret_cast<uintptr_t>(p->mixed) | reinterpret_cast<uintptr_t>(p->o) | reinterpret_cast<uintptr_t>(p->coef)) & 15))
    return 1006;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long warps = (long long)p->B * p->groups * p->KH;
  launch_pdl(delta_pairs_mma_kernel, dim3(unsigned((warps + 3) / 4)), dim3(128), 0, s, *p);
  const dim3 grid((p->vdim + DM_COLS - 1) / DM_COLS, p->H, p->B);
  if (p->dim <= 64) launch_pdl(delta_scan_mma_kernel<64>, grid, dim3(128), 0, s, *p);
  else launch_pdl(delta_scan_mma_kernel<128>, grid, dim3(128), 0, s, *p);
  return int(cudaGetLastError());
}
