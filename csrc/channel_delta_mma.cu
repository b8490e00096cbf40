// Gated delta rule with one decay per state row (channel_delta.cu has the recurrence): portions of a prompt on the tensor cores, bf16 rows of up to 128
// state rows
//
// The form of delta_rule_mma.cu: groups of DM = 16 tokens, the state in registers as the accumulator tiles of S^T, a warp for 16 value columns.  With
// P_i = g_1 .. g_i per row,
//
//   U = T (V - (P K) S),   O = (P Q) S + R U,   S <- diag(P_C) S + (K g_{j+1} .. g_C)^T U
//
// The decayed rows are fp32: channel_pairs_mma writes them as three bf16 pieces each (delta_mma.cuh), so the three products with the state are six
// tensor-core products each.  What it writes per group and head is the image of a stage of the scan's shared memory (rows swizzled for ldmatrix), which
// one bulk copy brings there.  Decay products are running products of factors in (0, 1], as in channel_delta.cu; the products of a key of the first
// eight tokens with a later one factor at the eighth token, so that only the two 8 x 8 blocks on the diagonal are summed pair by pair.
//
// Bounded like delta_rule_mma.cu; 350 MMAs a group and warp.  Scan and pairs, us, fp32 FMA form (channel_delta.cu) / this one, 128 x 128 states: 8 sequences of
// 2,048 tokens, 16 heads 1,213 / 847, 12 of 1,000 934 / 640, 3 of 1,501 537 / 327, one of 2,048 542 / 367, one of 512, 8 heads 121 / 99, one of 64 30 / 29.
// State against 64 bits: 0.84 to 0.995 of the FMA form's error on average (slow decays 1.2e-6 to 2.5e-6, the errors of the decays' exponentials; fast ones 0.5e-7).
#include "delta_mma.cuh"

namespace ats {

namespace {

constexpr int CM = 16;                   // tokens per group
constexpr int CM_B = 3 * 32 * 16;        // bytes of a 16 x 16 matrix as split B operand
constexpr int CM_COLS = 64;              // value columns of a CTA
constexpr int CM_STAGES = 2;
constexpr int CM_ROWS = 3 * CM;          // P k, P q, k g_{j+1} .. g_C

// Bytes per group and head: three pieces of the rows, T without its diagonal, R, P_C, the diagonal (the step sizes).
__host__ __device__ constexpr int cm_t_at(int DK) { return 3 * CM_ROWS * DK * 2; }
__host__ __device__ constexpr int cm_p_at(int DK) { return cm_t_at(DK) + 2 * CM_B; }
__host__ __device__ constexpr int cm_bytes(int DK) { return cm_p_at(DK) + DK * 4 + CM * 4; }
// Byte of channel d (even) of a row: 16-byte pieces exchanged inside 128 bytes by the row's last three bits.
__host__ __device__ constexpr int cm_at(int row, int d, int DK) { return row * DK * 2 + ((d >> 3 & ~7) | ((d >> 3 ^ row) & 7)) * 16 + (d & 7) * 2; }
constexpr int CM_PITCH = 132;            // floats of a row that the off-diagonal block is computed from
// Per group: 8 + 8 + 8 rows, the decays of the halves, kk (later T), kq (later R).
constexpr int CM_PAIR_FLOATS = 24 * CM_PITCH + 2 * 128 + 2 * CM * 17;

// Two warps per (group, head, sequence), one for each eight tokens, two channels per lane side by side.
template <int DK>
__global__ void __launch_bounds__(128, 3) channel_pairs_mma_kernel(const ChannelArgs p) {
  pdl_prologue();
  extern __shared__ __align__(16) float s_pair[];
  const int pair = threadIdx.x >> 6, half = threadIdx.x >> 5 & 1, lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
  const long long w = blockIdx.x * 2ll + pair;
  if (w >= (long long)p.B * p.groups * p.H) return;   // both warps of a pair; only barriers of the pair below
  const int h = int(w % p.H), grp = int((w / p.H) % p.groups), b = int(w / p.H / p.groups), kh = h / (p.H / p.KH);
  float* s_rows = s_pair + pair * CM_PAIR_FLOATS;      // 0..7 k of the second half, 8..15 q of it, 16..23 k of the first half, decayed inside their half
  float* s_decay = s_rows + 24 * CM_PITCH;             // [half][128]
  float(*s_kk)[17] = reinterpret_cast<float(*)[17]>(s_decay + 256);
  float(*s_kq)[17] = s_kk + CM;
  auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory"); };
  uint8_t* co = reinterpret_cast<uint8_t*>(p.coef) + w * cm_bytes(DK);
  const float rate = p.neg_rate[h];
  for (int i = threadIdx.x & 63; i < 2 * CM * 17; i += 64) s_kk[0][i] = 0.f;
  meet();
  auto put = [&](int row, int d, float x, float y) {
    uint32_t hi, mid, lo;
    split_pair(x, y, hi, mid, lo);
    uint8_t* at = co + cm_at(row, d, DK);
    *reinterpret_cast<uint32_t*>(at) = hi;
    *reinterpret_cast<uint32_t*>(at + CM_ROWS * DK * 2) = mid;
    *reinterpret_cast<uint32_t*>(at + 2 * CM_ROWS * DK * 2) = lo;
  };
  const int t0 = grp * CM + 8 * half, n = max(0, min(8, p.L - t0));
  const long long row0 = (long long)b * p.L + t0;
  {
    const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(p.mixed) + row0 * p.ldm + (long long)kh * p.dim;
    const __nv_bfloat16* k = q + (long long)p.KH * p.dim;
    const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(p.a) + row0 * p.lda + (long long)h * p.dim;
    const float* rl = p.rlen + row0 * 2 * p.KH;
    // sums[8 i + j]: i >= j: kq_ij; i < j: kk_ji
    float sums[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) sums[i] = 0.f;
#pragma unroll 1
    for (int d0 = lane * 2; d0 < DK; d0 += 64) {
      auto fetch = [&](const __nv_bfloat16* src, bool in) -> uint32_t { return in && d0 < p.dim ? *reinterpret_cast<const uint32_t*>(src + d0) : 0; };
      uint32_t pk[8], pq[8], pa[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        pk[i] = fetch(k + i * p.ldm, i < n);
        pq[i] = fetch(q + i * p.ldm, i < n);
        pa[i] = fetch(a + i * p.lda, i < n);
      }
      float dt[2], kv[8][2], qv[8][2], g[8][2], P[2] = {1.f, 1.f};
#pragma unroll
      for (int c = 0; c < 2; ++c) dt[c] = d0 + c < p.dim ? p.dt_bias[(long long)h * p.dim + d0 + c] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float rk = i < n ? rl[(long long)i * 2 * p.KH + p.KH + kh] : 0.f, rq = i < n ? rl[(long long)i * 2 * p.KH + kh] : 0.f;
        const float2 fk = unpack_bf16x2(pk[i]), fq = unpack_bf16x2(pq[i]), fa = unpack_bf16x2(pa[i]);
        kv[i][0] = fk.x * rk, kv[i][1] = fk.y * rk; qv[i][0] = fq.x * rq, qv[i][1] = fq.y * rq;
        g[i][0] = i < n && d0 < p.dim ? decay_of<__nv_bfloat16>(fa.x + dt[0], rate) : 1.f;
        g[i][1] = i < n && d0 + 1 < p.dim ? decay_of<__nv_bfloat16>(fa.y + dt[1], rate) : 1.f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        P[0] *= g[i][0], P[1] *= g[i][1];
        const float2 x = make_float2(kv[i][0] * P[0], kv[i][1] * P[1]), y = make_float2(qv[i][0] * P[0], qv[i][1] * P[1]);
        if (half == 0) {
          put(i, d0, x.x, x.y);
          put(CM + i, d0, y.x, y.y);
        } else {
          *reinterpret_cast<float2*>(s_rows + i * CM_PITCH + d0) = x;
          *reinterpret_cast<float2*>(s_rows + (8 + i) * CM_PITCH + d0) = y;
        }
      }
      *reinterpret_cast<float2*>(s_decay + half * 128 + d0) = make_float2(P[0], P[1]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float r[2] = {kv[j][0], kv[j][1]};
#pragma unroll
        for (int c = 0; c < 2; ++c) sums[j * 8 + j] += qv[j][c] * r[c];
#pragma unroll
        for (int i = j + 1; i < 8; ++i)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            r[c] *= g[i][c];
            sums[i * 8 + j] += qv[i][c] * r[c];
            sums[j * 8 + i] += kv[i][c] * r[c];
          }
        if (half == 0) *reinterpret_cast<float2*>(s_rows + (16 + j) * CM_PITCH + d0) = make_float2(r[0], r[1]);
        else put(2 * CM + 8 + j, d0, r[0], r[1]);
      }
    }
    // transposing reduction: after the steps, lane l holds the sums 2 l and 2 l + 1 over all lanes
#pragma unroll
    for (int i = 0; i < 32; ++i) sums[i] = keep_add(sums[i], sums[i + 32], lane, 16);
#pragma unroll
    for (int i = 0; i < 16; ++i) sums[i] = keep_add(sums[i], sums[i + 16], lane, 8);
#pragma unroll
    for (int i = 0; i < 8; ++i) sums[i] = keep_add(sums[i], sums[i + 8], lane, 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) sums[i] = keep_add(sums[i], sums[i + 4], lane, 2);
#pragma unroll
    for (int i = 0; i < 2; ++i) sums[i] = keep_add(sums[i], sums[i + 2], lane, 1);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = g8, j = 2 * t + e;
      if (i >= j) s_kq[8 * half + i][8 * half + j] = sums[e];
      else s_kk[8 * half + j][8 * half + i] = sums[e];
    }
  }
  meet();
  // the rows that the other half decays further
#pragma unroll 1
  for (int d0 = lane * 2; d0 < DK; d0 += 64) {
    const float2 P = *reinterpret_cast<const float2*>(s_decay + (1 - half) * 128 + d0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (half == 0) {
        const float2 x = *reinterpret_cast<const float2*>(s_rows + (16 + i) * CM_PITCH + d0);
        put(2 * CM + i, d0, x.x * P.x, x.y * P.y);
      } else {
        const float2 x = *reinterpret_cast<const float2*>(s_rows + i * CM_PITCH + d0), y = *reinterpret_cast<const float2*>(s_rows + (8 + i) * CM_PITCH + d0);
        put(8 + i, d0, x.x * P.x, x.y * P.y);
        put(CM + 8 + i, d0, y.x * P.x, y.y * P.y);
      }
    }
    if (half == 0) {
      const float2 mine = *reinterpret_cast<const float2*>(s_decay + d0);
      *reinterpret_cast<float2*>(co + cm_p_at(DK) + d0 * 4) = make_float2(mine.x * P.x, mine.y * P.y);
    }
  }
  if (half == 0) {   // second half against the first: rows k and q of one A operand
    float big[4] = {}, small[4] = {};
#pragma unroll 2
    for (int s = 0; s < DK / 16; ++s) {
      uint32_t a[3][4], bb[3][2];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 v = *reinterpret_cast<const float2*>(s_rows + (g8 + 8 * (x & 1)) * CM_PITCH + s * 16 + 8 * (x >> 1) + 2 * t);
        split_pair(v.x, v.y, a[0][x], a[1][x], a[2][x]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 v = *reinterpret_cast<const float2*>(s_rows + (16 + g8) * CM_PITCH + s * 16 + 8 * x + 2 * t);
        split_pair(v.x, v.y, bb[0][x], bb[1][x], bb[2][x]);
      }
      mma_bf16(big, a[0], bb[0][0], bb[0][1]);
      mma_bf16(small, a[2], bb[0][0], bb[0][1]);
      mma_bf16(small, a[0], bb[2][0], bb[2][1]);
      mma_bf16(small, a[1], bb[1][0], bb[1][1]);
      mma_bf16(small, a[1], bb[0][0], bb[0][1]);
      mma_bf16(small, a[0], bb[1][0], bb[1][1]);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      s_kk[8 + g8][2 * t + e] = big[e] + small[e];
      s_kq[8 + g8][2 * t + e] = big[2 + e] + small[2 + e];
    }
    __syncwarp();
    float y[CM], bc = 0.f;
    if (lane < CM) {   // lane = column of the inverse, by forward substitution; times the column's step size
      const int tokens = min(CM, p.L - grp * CM);
      const float* gb = p.gb + row0 * 2 * p.H + p.H + h;
      float beta[CM];
#pragma unroll
      for (int i = 0; i < CM; ++i) {
        beta[i] = i < tokens ? gb[(long long)i * 2 * p.H] : 0.f;
        if (i == lane) bc = beta[i];
      }
#pragma unroll
      for (int i = 0; i < CM; ++i) {
        float acc = i == lane ? 1.f : 0.f;
#pragma unroll
        for (int j = i - 1; j >= 0; --j) acc -= beta[i] * s_kk[i][j] * y[j];
        y[i] = acc;
      }
    }
    __syncwarp();
    if (lane < CM) {
#pragma unroll
      for (int i = 0; i < CM; ++i) s_kk[i][lane] = i <= lane ? 0.f : y[i] * bc;   // T
      reinterpret_cast<float*>(co + cm_p_at(DK))[DK + lane] = bc;
    }
    __syncwarp();
    store_split_b(s_kk, lane, reinterpret_cast<uint4*>(co + cm_t_at(DK)));
  }
  meet();
  if (half == 1) store_split_b(s_kq, lane, reinterpret_cast<uint4*>(co + cm_t_at(DK) + CM_B));
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, int bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

template <int DK>
__global__ void __launch_bounds__(128, 2) channel_scan_mma_kernel(const ChannelArgs p, int* status) {
  pdl_prologue();
  constexpr int NT = DK / 8, KS = DK / 16, VPITCH = CM_COLS * 2 + 16, V_AT = cm_bytes(DK), STAGE = V_AT + CM * VPITCH, PIECE = CM_ROWS * DK * 2;
  constexpr int OPITCH = 48;
  extern __shared__ __align__(16) uint8_t s_ring[];   // [CM_STAGES][STAGE]
  __shared__ __align__(16) uint8_t s_out[4][CM * OPITCH];
  __shared__ uint64_t s_full[CM_STAGES];
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int h = blockIdx.y, b = blockIdx.z;
  const int cta0 = blockIdx.x * CM_COLS, col0 = cta0 + warp * 16;
  if (tid == 0) {
    for (int i = 0; i < CM_STAGES; ++i) mbar_init(&s_full[i], 1);
    s_abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  float S[NT][4];   // tile j: rows = columns col0 + g (+ 8) of the state, columns = its rows 8 j + 2 t, + 1
  float* st = p.state + (long long)b * p.state_bs + (long long)h * p.dim * p.vdim;
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * j + 2 * t + (e & 1), col = col0 + g + 8 * (e >> 1);
      S[j][e] = !p.fresh && d < p.dim && col < p.vdim ? st[(long long)d * p.vdim + col] : 0.f;
    }
  const __nv_bfloat16* vbase = static_cast<const __nv_bfloat16*>(p.mixed) + (long long)b * p.L * p.ldm + 2 * p.KH * p.dim + (long long)h * p.vdim + cta0;
  const uint8_t* cbase = reinterpret_cast<const uint8_t*>(p.coef) + ((long long)b * p.groups * p.H + h) * cm_bytes(DK);
  auto request = [&](int grp) {   // the stage is read by nobody any more
    if (grp >= p.groups) return;
    uint8_t* stage = s_ring + (grp % CM_STAGES) * STAGE;
    const int t0 = grp * CM, n = min(CM, p.L - t0);
    if (tid == 0) {
      mbar_expect_tx(&s_full[grp % CM_STAGES], cm_bytes(DK));
      bulk_load(smem_u32(stage), cbase + (long long)grp * p.H * cm_bytes(DK), cm_bytes(DK), &s_full[grp % CM_STAGES]);
    }
    const int tok = tid >> 3, c = (tid & 7) * 8;
    const bool in = tok < n && cta0 + c < p.vdim;
    cp_async_fill(smem_u32(stage) + V_AT + tok * VPITCH + c * 2, in ? vbase + (long long)(t0 + tok) * p.ldm + c : static_cast<const __nv_bfloat16*>(p.mixed), in ? 16 : 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  request(0);
  // ldmatrix: lane l points at row l % 8 of block l / 8; see delta_rule_mma.cu
  const int prow = (lane & 7) + (lane >> 4) * 8, ppiece = lane >> 3 & 1, trow = (lane & 7) + (lane >> 3 & 1) * 8, tpiece = lane >> 4;
  const uint32_t vturned = uint32_t(trow * VPITCH + tpiece * 16 + warp * 32);
  const uint32_t out_at = smem_u32(s_out[warp]);
  bool ok = true;
  for (int grp = 0; grp < p.groups; ++grp) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    ok = mbar_wait_bounded(&s_full[grp % CM_STAGES], (grp / CM_STAGES) & 1, &s_abort, status, kTimeoutFull);
    if (!__syncthreads_and(ok)) break;   // this group's rows are there for everyone, and everyone is done with the group before
    request(grp + 1);
    const uint8_t* stage = s_ring + (grp % CM_STAGES) * STAGE;
    const uint32_t at = smem_u32(stage);
    const uint4* mt = reinterpret_cast<const uint4*>(stage + cm_t_at(DK));
    const uint4* mr = reinterpret_cast<const uint4*>(stage + cm_t_at(DK) + CM_B);
    const float* decay = reinterpret_cast<const float*>(stage + cm_p_at(DK));
    const int t0 = grp * CM, n = min(CM, p.L - t0);
    float sk[2][4] = {}, sq[2][4] = {}, ek[2][4] = {}, eq[2][4] = {};   // [column][token]; the leading pieces apart from the others
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      Pieces a;
      split_tiles(S[2 * s], S[2 * s + 1], a);
      const uint32_t kat = at + cm_at(prow, 16 * s + 8 * ppiece, DK), qat = at + cm_at(CM + prow, 16 * s + 8 * ppiece, DK);
      uint32_t kb[4], qb[4];
      ldsm4(kb, kat);
      ldsm4(qb, qat);
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
      ldsm4(kb, kat + 2 * PIECE);
      ldsm4(qb, qat + 2 * PIECE);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mma_bf16(ek[x], a.hi, kb[2 * x], kb[2 * x + 1]);
        mma_bf16(eq[x], a.hi, qb[2 * x], qb[2 * x + 1]);
      }
      ldsm4(kb, kat + PIECE);
      ldsm4(qb, qat + PIECE);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mma_bf16(ek[x], a.mid, kb[2 * x], kb[2 * x + 1]);
        mma_bf16(eq[x], a.mid, qb[2 * x], qb[2 * x + 1]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mma_bf16(ek[x], a.hi, kb[2 * x], kb[2 * x + 1]);
        mma_bf16(eq[x], a.hi, qb[2 * x], qb[2 * x + 1]);
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
        const float2 lo = unpack_bf16x2(vv[x]), hi = unpack_bf16x2(vv[2 + x]);
        sk[x][0] = lo.x - (sk[x][0] + ek[x][0]);
        sk[x][1] = lo.y - (sk[x][1] + ek[x][1]);
        sk[x][2] = hi.x - (sk[x][2] + ek[x][2]);
        sk[x][3] = hi.y - (sk[x][3] + ek[x][3]);
      }
      spoilt = solve_group(sk, mt, decay + DK, lane, u, eu, first);
    }
    split_tiles(u[0], u[1], eu[0], eu[1], a);
#pragma unroll
    for (int s = 0; s < KS; ++s) {   // the state first: the next group waits for it
      const uint32_t kat = at + cm_at(2 * CM + trow, 16 * s + 8 * tpiece, DK);
      uint32_t kh[4], km[4], kl[4];
      ldsm4_t(kh, kat);
      ldsm4_t(km, kat + PIECE);
      ldsm4_t(kl, kat + 2 * PIECE);
      float d[2][4] = {}, f[2][4] = {};
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mma_bf16(d[x], a.hi, kh[2 * x], kh[2 * x + 1]);
        mma_bf16(f[x], a.lo, kh[2 * x], kh[2 * x + 1]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) mma_bf16(f[x], a.hi, kl[2 * x], kl[2 * x + 1]);
#pragma unroll
      for (int x = 0; x < 2; ++x) mma_bf16(f[x], a.mid, km[2 * x], km[2 * x + 1]);
#pragma unroll
      for (int x = 0; x < 2; ++x) mma_bf16(f[x], a.mid, kh[2 * x], kh[2 * x + 1]);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mma_bf16(f[x], a.hi, km[2 * x], km[2 * x + 1]);
        add_rest(d[x], f[x], a.hi, kh[2 * x], kh[2 * x + 1]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 P = *reinterpret_cast<const float2*>(decay + 16 * s + 8 * x + 2 * t);
        float(&S_)[4] = S[2 * s + x];
        S_[0] = fmaf(S_[0], P.x, f[x][0]) + d[x][0];
        S_[1] = fmaf(S_[1], P.y, f[x][1]) + d[x][1];
        S_[2] = fmaf(S_[2], P.x, f[x][2]) + d[x][2];
        S_[3] = fmaf(S_[3], P.y, f[x][3]) + d[x][3];
      }
    }
    {
      float o[2][4];
      split_product(a, mr, lane, o);
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[x][e] += sq[x][e] + eq[x][e];
      if (spoilt) {
        spoil(o, t, first);
        spoil_state(S, first);
      }
      // [token][column] in shared memory: blocks (tokens 0..7, columns 0..7), (0..7, 8..15), (8..15, 0..7), (8..15, 8..15)
      stsm4_t(out_at + prow * OPITCH + ppiece * 16, pack_bf16x2(o[0][0], o[0][1]), pack_bf16x2(o[0][2], o[0][3]), pack_bf16x2(o[1][0], o[1][1]),
              pack_bf16x2(o[1][2], o[1][3]));
      __syncwarp();
      const int tok = lane >> 1, col = col0 + (lane & 1) * 8;
      const uint4 v = *reinterpret_cast<const uint4*>(s_out[warp] + tok * OPITCH + (lane & 1) * 16);
      if (tok < n && col < p.vdim)
        *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.o) + ((long long)b * p.L + t0 + tok) * p.ldo + (long long)h * p.vdim + col) = v;
      __syncwarp();
    }
  }
  if (!ok) {   // a copy that was issued lands before the CTA gives its shared memory back
    const uint64_t from = globaltimer_ns();
    while (globaltimer_ns() - from < 10000000ull) {
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

template <int DK>
int launch_channel_mma(const ChannelArgs& p, int* status, cudaStream_t s) {
  const int pair_smem = 2 * CM_PAIR_FLOATS * int(sizeof(float)), scan_smem = CM_STAGES * (cm_bytes(DK) + CM * (CM_COLS * 2 + 16));
  auto pairs = channel_pairs_mma_kernel<DK>;
  if (cudaError_t e = cudaFuncSetAttribute(pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem)) return int(e);
  if (cudaError_t e = cudaFuncSetAttribute(channel_scan_mma_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, scan_smem)) return int(e);
  const long long groups = (long long)p.B * p.groups * p.H;
  launch_pdl(pairs, dim3(unsigned((groups + 1) / 2)), dim3(128), size_t(pair_smem), s, p);
  launch_pdl(channel_scan_mma_kernel<DK>, dim3((p.vdim + CM_COLS - 1) / CM_COLS, p.H, p.B), dim3(128), size_t(scan_smem), s, p, status);
  return int(cudaGetLastError());
}

}  // namespace
}  // namespace ats

using namespace ats;

// bf16 rows whose values are whole 16-byte pieces (dim, vdim, ldm, ldo multiples of 8, mixed and o 16-byte aligned; decay inputs in pairs), dim up to DK (64 or 128), p->groups
// groups of 16 tokens; coef: per (sequence, group, head) 292 DK + 3136 bytes (cm_bytes), 16-byte aligned.
ATS_API int ats_channel_delta_mma(const ChannelArgs* p, int* status, void* stream) {
  if (p->B <= 0 || p->L <= 0) return 0;
  if (p->groups != (p->L + CM - 1) / CM || p->KH < 1 || p->H % p->KH || (p->DK != 64 && p->DK != 128) || p->dim < 1 || p->dim > p->DK ||
      ((p->dim | p->vdim | p->ldm | p->ldo) & 7) || (p->lda & 1) || (reinterpret_cast<uintptr_t>(p->a) & 3) || ((reinterpret_cast<uintptr_t>(p->mixed) | reinterpret_cast<uintptr_t>(p->o) | reinterpret_cast<uintptr_t>(p->coef)) & 15))
    return 1006;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return p->DK == 64 ? launch_channel_mma<64>(*p, status, s) : launch_channel_mma<128>(*p, status, s);
}
