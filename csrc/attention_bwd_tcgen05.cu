// Causal grouped-query flash attention backward for sm_100a on tcgen05 tensor cores.
//
// Two passes share one kernel template (plus a tiny pre-pass delta = rowsum(dO * O)):
//   MODE 0 (dK, dV): one CTA per (128-key tile j, kv head, batch).  K_j and V_j stay in shared memory; for every query
//           head of the group and every query tile i >= j the CTA streams Q_i and dO_i, recomputes S = Q K^T and
//           dP = dO V^T on the tensor cores, forms P = exp(S - lse) and dS = P * (dP - delta) * scale in registers, and
//           accumulates dV += P^T dO and dK += dS^T Q in TMEM across all iterations (no atomics, deterministic).
//   MODE 1 (dQ):     one CTA per (128-query tile i, query head, batch).  Q_i and dO_i stay resident, K_j / V_j stream for
//           j <= i, and dQ += dS K accumulates in TMEM; dS goes back to tensor memory as bf16 and is the MMA's A operand.
// S and dP are recomputed in both passes (7 tile products per tile pair instead of 5) in exchange for an atomics-free,
// deterministic dQ.
//
// The dK/dV pass needs P^T and dS^T as A operands.
//   64 dimensions:  P and dS go to shared memory as [query x key] bf16 tiles in the 128-byte-swizzled layout, which the same bytes serve as an
//           MN-major operand.
//   128 dimensions (OVER): those tiles would take the room of a second stage, and copies, products and exponentials would follow one another
//           (568 us for one sequence of 4,096 tokens, 32 / 8 heads).  So the scores are computed transposed, S^T = K Q^T and dP^T = V dO^T, with keys
//           as the lanes of tensor memory: P^T and dS^T are written over the scores they come from and are read from there.  The scores of pair t + 1
//           run under dS of pair t, dP of t + 1 under the exponentials of t + 1: 263 us.  At 64 dimensions that form is the slower one (579 us
//           for 8 x 2,048 tokens, 32 / 4 heads, where the other takes 397): products with an A operand in tensor memory and 64 columns take longer than
//           from shared memory, and the statistics of a query are read per column.
// In the other forms the scores of pair t + 1 run as soon as S of pair t is in registers, dP of t + 1 as soon as dP of t is.
//
//   warp 0: TMA producer   warp 1: TMEM owner + MMA issuer   warps 2..9: two threads per row of the scores (64 columns each)
// Any sequence length: rows behind the end of a sequence read as zero (its length is a dimension of the tensor maps).  Queries there get a
// log-sum-exp of infinity, so their P and dS vanish; keys there are behind every real query; neither is stored.
// Every wait is bounded (status word + clean unwind); no load uses cluster multicast.
//
// Replaces the flash-attn / SDPA backward the reference relies on (reference core/model.py:763-768).
#include "common.cuh"

namespace ats {

int make_tmap_batched(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t batch, uint64_t ld, uint64_t batch_stride, uint32_t box_rows);

constexpr int AB_SPLIT = 2;                       // threads per row of the scores in the softmax-gradient stage
constexpr int AB_COLS = 128 / AB_SPLIT;           // columns per thread
constexpr int AB_THREADS = 64 + 128 * AB_SPLIT;   // TMA warp, MMA warp, 4 * AB_SPLIT softmax-gradient warps

struct AttnBwdArgs {
  int B, L, Hq, Hkv, D;
  int q_col0, k_col0, v_col0;
  const float* lse;    // [B, Hq, L] natural log
  const float* delta;  // [B, Hq, L]
  __nv_bfloat16* dq;   // row = token, pitch ld_dq elements, head h at column h * D
  __nv_bfloat16* dk;   // row = token, pitch ld_dkv
  __nv_bfloat16* dv;
  long long ld_dq, ld_dkv;
  float scale, scale_log2;
  int* status;
  long long* prof;  // optional [16]: cycle totals, written by one CTA (diagnostics; null in normal use)
};

enum : int { kNone, kAll, kDiagonal };
template <int V> struct Masks { static constexpr int value = V; };

// FORM 1: MODE 0 at 128 dimensions where each CTA has one pair of tiles (up to 128 tokens, no shared keys): there is nothing to run ahead of, and the form of 64
// dimensions ends sooner (8 heads of 100 tokens 7.3 us, OVER 8.0); MODE 1 for more than eight tiles: see MASKS.
template <int D, int MODE, int FORM>
struct AttnBwdSmem {
  // streamed stages: a stage is held until the gradient products that read it have finished, and a refill takes a
  // TMA round trip, so the ring must be deep enough to have the next tiles in flight meanwhile
  static constexpr int ST = (D == 64) ? 4 : (MODE == 0 && FORM == 1) ? 1 : 2;
  static constexpr int TB = 128 * D * 2;
  static constexpr int R1 = 0, R2 = TB;
  static constexpr int T1 = 2 * TB;            // ST stages
  static constexpr int T2 = T1 + ST * TB;      // ST stages
  static constexpr bool OVER = MODE == 0 && D == 128 && FORM == 0;
  static constexpr int P_OFF = T2 + ST * TB;     // MODE 0 at 64 dimensions: P, dS
  static constexpr int DS_OFF = P_OFF + (MODE == 0 && !OVER ? 32768 : 0);
  static constexpr int ROW_OFF = DS_OFF + (MODE == 0 && !OVER ? 32768 : 0);   // OVER: [2][-lse, -delta][128 queries] of two iterations
  static constexpr int BAR_OFF = ROW_OFF + (OVER ? 2048 : 0);
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

// delta[b, h, i] = sum_d dO[b, i, h, d] * O[b, i, h, d].  Eight elements (16 bytes) per thread, D / 8 threads per row, so a
// warp covers 32 / (D / 8) rows with fully coalesced 512-byte accesses.
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                                                         float* __restrict__ delta, int B, int L, int Hq, int D) {
  const int tpr = D >> 3;  // threads per row: 8 (D = 64) or 16 (D = 128)
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long row = g / tpr;  // (token, head) row
  const int part = int(g % tpr);
  const long long total = (long long)B * L * Hq;
  float acc = 0.f;
  if (row < total) {
    const uint4 a = reinterpret_cast<const uint4*>(dout + row * D)[part];
    const uint4 o = reinterpret_cast<const uint4*>(out + row * D)[part];
    const float2 a0 = unpack_bf16x2(a.x), a1 = unpack_bf16x2(a.y), a2 = unpack_bf16x2(a.z), a3 = unpack_bf16x2(a.w);
    const float2 o0 = unpack_bf16x2(o.x), o1 = unpack_bf16x2(o.y), o2 = unpack_bf16x2(o.z), o3 = unpack_bf16x2(o.w);
    acc = a0.x * o0.x + a0.y * o0.y + a1.x * o1.x + a1.y * o1.y + a2.x * o2.x + a2.y * o2.y + a3.x * o3.x + a3.y * o3.y;
  }
  for (int off = tpr >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (row < total && part == 0) {
    const int h = int(row % Hq);
    const long long tok = row / Hq;
    const int b = int(tok / L), i = int(tok % L);
    delta[((long long)b * Hq + h) * L + i] = acc;
  }
}

template <int D, int MODE, int FORM>
__global__ void __launch_bounds__(AB_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do, const AttnBwdArgs p) {
  using SM = AttnBwdSmem<D, MODE, FORM>;
  constexpr int ST = SM::ST;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sR1 = smem + SM::R1;
  uint8_t* sR2 = smem + SM::R2;
  uint8_t* sT1 = smem + SM::T1;
  uint8_t* sT2 = smem + SM::T2;
  uint8_t* sP = smem + SM::P_OFF;
  uint8_t* sDS = smem + SM::DS_OFF;
  float* sRow = reinterpret_cast<float*>(smem + SM::ROW_OFF);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::BAR_OFF);
  uint64_t* res_full = bars;       // 1
  uint64_t* t_full = bars + 1;     // [4]
  uint64_t* t_empty = bars + 5;    // [4]
  uint64_t* s_full = bars + 9;     // S ready
  uint64_t* dp_full = bars + 10;   // dP ready
  uint64_t* s_free = bars + 11;    // one arrival per softmax warp: S read out of TMEM
  uint64_t* dp_free = bars + 12;   // the same for dP
  uint64_t* p_full = bars + 13;    // OVER: one arrival per softmax warp, P written to TMEM
  uint64_t* ds_full = bars + 14;   // the same for dS (VIA_SMEM: P and dS written to shared memory)
  uint64_t* ds_free = bars + 15;   // without OVER: the products that read P and dS are done
  uint64_t* acc_done = bars + 16;
  uint64_t* row_full = bars + 17;  // OVER: one arrival per softmax warp, its share of an iteration's statistics written and those before read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (p.L + 127) / 128;
  const int rep = p.Hq / p.Hkv;
  // Grid = (heads, batch, tiles): CTAs are handed out x-fastest, so with the tile index slowest every CTA of the heaviest
  // tile (of all heads and sequences) starts before any lighter one.  With the tile index fastest, a heavy tile of the
  // last heads started late and the causal imbalance left SMs idle for a quarter of the dK/dV pass.
  const int b = blockIdx.y;
  // fixed tile of this CTA and iteration space
  int fixed, head, n_iter;
  if (MODE == 0) {
    fixed = blockIdx.z;  // key tile j (j = 0 has the most work)
    head = blockIdx.x;   // kv head
    n_iter = rep * (nq - fixed);
  } else {
    fixed = nq - 1 - blockIdx.z;  // query tile i (the last one has the most work)
    head = blockIdx.x;            // query head
    n_iter = fixed + 1;
  }
  const int hk = MODE == 0 ? head : head / rep;

  if (threadIdx.x == 0) {
    mbar_init(res_full, 1);
    for (int s = 0; s < 4; ++s) {
      mbar_init(&t_full[s], 1);
      mbar_init(&t_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(s_free, 4 * AB_SPLIT);
    mbar_init(dp_free, 4 * AB_SPLIT);
    mbar_init(p_full, 4 * AB_SPLIT);
    mbar_init(ds_full, 4 * AB_SPLIT);
    mbar_init(ds_free, 1);
    mbar_init(acc_done, 1);
    mbar_init(row_full, 4 * AB_SPLIT);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base, tmem_dP = tmem_base + 128, tmem_A1 = tmem_base + 256, tmem_A2 = tmem_base + 256 + D;
  // OVER: P and dS as bf16 pairs over the scores that their thread has read, so the second half of the columns starts 64 further on.  MODE 1: dS
  // in 64 columns of its own.
  constexpr bool OVER = SM::OVER, VIA_SMEM = MODE == 0 && !OVER;
  const uint32_t tmem_P = tmem_S, tmem_dS = OVER ? tmem_dP : tmem_base + 384;
  // Masks of the pair on the diagonal: in every iteration where that is a large share of them (dQ of up to eight tiles: 8 x 384 tokens, 32 / 8 heads 32.3 us,
  // two loops 33.5), else one loop with them and one without (one sequence of 4,096: 161 and 154).
  constexpr int MASKS = MODE == 0 ? (FORM == 1 ? kAll : kNone) : (FORM == 0 ? kDiagonal : kNone);
  constexpr uint32_t HALF = OVER ? 64 : 32;   // columns from the first 64 reduction elements to the others

  // iteration t -> (query head, query tile, key tile)
  auto decode = [&](int t, int& h, int& qi, int& kj) {
    if (MODE == 0) {
      const int per = nq - fixed;
      h = head * rep + t / per;
      qi = fixed + t % per;
      kj = fixed;
    } else {
      h = head;
      qi = fixed;
      kj = t;
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------------------ producer
      mbar_expect_tx(res_full, 2 * SM::TB);
      if (MODE == 0) {
        const int row = fixed * 128;
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          tma_load_3d(sR1 + c * 16384, &map_k, res_full, p.k_col0 + hk * D + 64 * c, row, b);
          tma_load_3d(sR2 + c * 16384, &map_v, res_full, p.v_col0 + hk * D + 64 * c, row, b);
        }
      } else {
        const int row = fixed * 128;
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          tma_load_3d(sR1 + c * 16384, &map_q, res_full, p.q_col0 + head * D + 64 * c, row, b);
          tma_load_3d(sR2 + c * 16384, &map_do, res_full, head * D + 64 * c, row, b);
        }
      }
      for (int t = 0; t < n_iter; ++t) {
        const int s = t % ST, ph = (t / ST) & 1;
        int h, qi, kj;
        decode(t, h, qi, kj);
        if (!mbar_wait_bounded(&t_empty[s], ph ^ 1, abort_flag, p.status, kTimeoutEmpty)) break;
        mbar_expect_tx(&t_full[s], 2 * SM::TB);
        if (MODE == 0) {
          const int row = qi * 128;
#pragma unroll
          for (int c = 0; c < D / 64; ++c) {
            tma_load_3d(sT1 + s * SM::TB + c * 16384, &map_q, &t_full[s], p.q_col0 + h * D + 64 * c, row, b);
            tma_load_3d(sT2 + s * SM::TB + c * 16384, &map_do, &t_full[s], h * D + 64 * c, row, b);
          }
        } else {
          const int row = kj * 128;
#pragma unroll
          for (int c = 0; c < D / 64; ++c) {
            tma_load_3d(sT1 + s * SM::TB + c * 16384, &map_k, &t_full[s], p.k_col0 + hk * D + 64 * c, row, b);
            tma_load_3d(sT2 + s * SM::TB + c * 16384, &map_v, &t_full[s], p.v_col0 + hk * D + 64 * c, row, b);
          }
        }
      }
      if (*abort_flag) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 20000ull) {
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ------------------------------------------------------------------ MMA issuer
      const uint32_t idesc_s = make_idesc(128, 128, 1, 1, 0, 0);
      const uint32_t idesc_acc = make_idesc(128, D, 1, 1, VIA_SMEM, 1);  // A from tensor memory or MN-major, B MN-major
      // Descriptors are built once: per operand one base descriptor for the K-major view and one for the MN-major view;
      // inside the loops a descriptor is the base plus a constant (the issue rate of this one thread bounds the kernel).
      const uint64_t r1_k = make_smem_desc_sw128(smem_u32(sR1), 16, 1024), r2_k = make_smem_desc_sw128(smem_u32(sR2), 16, 1024);
      const uint64_t t1_k = make_smem_desc_sw128(smem_u32(sT1), 16, 1024), t2_k = make_smem_desc_sw128(smem_u32(sT2), 16, 1024);
      const uint64_t t1_mn = make_smem_desc_sw128(smem_u32(sT1), 16384, 1024), t2_mn = make_smem_desc_sw128(smem_u32(sT2), 16384, 1024);
      const uint64_t p_mn = make_smem_desc_sw128(smem_u32(sP), 16384, 1024), ds_mn = make_smem_desc_sw128(smem_u32(sDS), 16384, 1024);
      // S (which = 0: R1 and T1) or dP (1: R2 and T2) of iteration t; lanes are the rows of the resident tile, VIA_SMEM: of the streamed one
      auto issue_score = [&](int t, int which) {
        const uint64_t fixed_d = which ? r2_k : r1_k, moving = desc_advance(which ? t2_k : t1_k, uint32_t(t % ST) * SM::TB);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k >> 2) * 16384 + (k & 3) * 32;
          const uint64_t f = desc_advance(fixed_d, off), m = desc_advance(moving, off);
          tc_mma_f16(which ? tmem_dP : tmem_S, VIA_SMEM ? m : f, VIA_SMEM ? f : m, idesc_s, k != 0);
        }
        tc_commit(which ? dp_full : s_full);
      };
      auto issue_acc = [&](int t, uint32_t acc, uint32_t a, uint64_t rows_mn) {   // reduction over the 128 rows of the streamed tile, 16 per step
        const uint64_t bb = desc_advance(rows_mn, uint32_t(t % ST) * SM::TB);
#pragma unroll
        for (int k = 0; k < 8; ++k) tc_mma_f16_ts(acc, a + (k >> 2) * HALF + (k & 3) * 8, desc_advance(bb, k * 2048), idesc_acc, (t | k) != 0);
      };
      auto issue_acc_smem = [&](int t, uint32_t acc, uint64_t a_mn, uint64_t rows_mn) {
        const uint64_t bb = desc_advance(rows_mn, uint32_t(t % ST) * SM::TB);
#pragma unroll
        for (int k = 0; k < 8; ++k) tc_mma_f16(acc, desc_advance(a_mn, k * 2048), desc_advance(bb, k * 2048), idesc_acc, (t | k) != 0);
      };
      long long waited = 0, c0 = 0;
      const bool rec = p.prof != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0;
      auto wait = [&](uint64_t* bar, int parity, int code) {
        if (rec) c0 = clock64();
        const bool got = mbar_wait_bounded(bar, parity, abort_flag, p.status, code);
        if (rec) waited += clock64() - c0;
        tc_fence_after();
        return got;
      };
      const long long t_begin = clock64();
      bool ok = wait(res_full, 0, kTimeoutFull) && (n_iter == 0 || wait(&t_full[0], 0, kTimeoutFull));
      if (ok && n_iter > 0) {
        issue_score(0, 0);
        issue_score(0, 1);
      }
      for (int t = 0; ok && t < n_iter; ++t) {
        const bool more = t + 1 < n_iter;
        auto next_scores = [&] {
          ok = ok && wait(&t_full[(t + 1) % ST], ((t + 1) / ST) & 1, kTimeoutFull) && (OVER || wait(s_free, t & 1, kTimeoutTmemEmpty));
          if (ok) issue_score(t + 1, 0);
        };
        auto next_dp = [&] {
          ok = ok && (OVER || wait(dp_free, t & 1, kTimeoutTmemEmpty));
          if (ok) issue_score(t + 1, 1);
        };
        if (OVER) {
          ok = ok && wait(p_full, t & 1, kTimeoutTmemFull);
          if (!ok) break;
          issue_acc(t, tmem_A1, tmem_P, t2_mn);   // dV += P^T dO
          if (more) next_scores();   // (products are executed in the order of their issue: P has been read when S is written)
        } else if (more) {
          next_scores();
          next_dp();
        }
        ok = ok && wait(ds_full, t & 1, kTimeoutTmemFull);
        if (!ok) break;
        if (VIA_SMEM) {
          issue_acc_smem(t, tmem_A1, p_mn, t2_mn);
          issue_acc_smem(t, tmem_A2, ds_mn, t1_mn);
        } else {
          issue_acc(t, MODE == 0 ? tmem_A2 : tmem_A1, tmem_dS, t1_mn);   // dK += dS^T Q, dQ += dS K
        }
        if (!OVER) tc_commit(ds_free);
        tc_commit(&t_empty[t % ST]);
        if (OVER && more) next_dp();
      }
      if (rec) {
        p.prof[0] = clock64() - t_begin;
        p.prof[1] = waited;
        p.prof[5] = n_iter;
      }
      tc_commit(acc_done);
    }
  } else {
    // ---------------------------------------- softmax-gradient threads: a TMEM lane quadrant is open to warps with the
    // same (warp % 4), so the AB_SPLIT warps w, w + 4, ... share 32 rows and take AB_COLS columns each
    const int quad = warp & 3;
    const int part = (warp - 2) >> 2;  // which AB_COLS key columns of the 128
    const int r = quad * 32 + lane;
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    bool ok = true;
    // Query tile and head of the next statistics to fetch (MODE 1: of all of them), and of the iteration at hand whether it is on the diagonal.
    int tile = fixed, stat_head = MODE == 0 ? head * rep : head, to_diagonal = 0;
    // log-sum-exp or delta of query `row` of that tile, as they are: what is multiplied here would be waited for here
    auto row_stat = [&](int row, bool lse) {
      const long long idx = ((long long)b * p.Hq + stat_head) * p.L + tile * 128 + row;
      const bool real = tile * 128 + row < p.L;
      return lse ? (real ? p.lse[idx] : INFINITY) : (real ? p.delta[idx] : 0.f);
    };
    auto scaled = [&](float v, bool lse) { return lse ? v * -1.4426950408889634f : -v * p.scale; };
    auto next_tile = [&] {
      if (++tile == nq) tile = fixed, ++stat_head;
    };
    // OVER: queries are the columns; each thread fetches one value an iteration ahead and leaves it in shared memory, where everyone reads it.
    // Otherwise they are the rows, and a thread fetches those of its row (VIA_SMEM: of the next iteration's row, ahead).
    const int id = int(threadIdx.x) - 64;
    float row_l = 0.f, row_d = 0.f, ahead = 0.f, ahead_d = 0.f;
    if (OVER) {
      if (n_iter > 0) sRow[id] = scaled(row_stat(id & 127, id < 128), id < 128);
      next_tile();
      if (n_iter > 1) ahead = row_stat(id & 127, id < 128);
    } else if (n_iter > 0) {
      row_l = ahead = row_stat(r, true), row_d = ahead_d = row_stat(r, false);
    }
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), scale2 = make_float2(p.scale, p.scale);
    const uint32_t col = lane_base + part * AB_COLS, bf_col = lane_base + part * HALF;
    for (int t = 0; t < n_iter; ++t) {
      const bool diag = MODE == 0 ? to_diagonal == 0 : t == n_iter - 1;
      if (MODE == 0 && ++to_diagonal == nq - fixed) to_diagonal = 0;
      const float* nl = sRow + (t & 1) * 256 + part * AB_COLS;   // of this thread's columns; 128 floats on those of delta
      if (OVER) {
        // The values of this iteration are there, those of the one before are read.  (No named barrier: a warp that has given up never comes to it.)
        __syncwarp();
        if (lane == 0) mbar_arrive(row_full);
        if (!mbar_wait_warp(row_full, t & 1, abort_flag, p.status, kTimeoutFull)) {
          ok = false;
          break;
        }
        if (t + 1 < n_iter) sRow[((t + 1) & 1) * 256 + id] = scaled(ahead, id < 128);
        next_tile();
        if (t + 2 < n_iter) ahead = row_stat(id & 127, id < 128);
      } else if (VIA_SMEM) {
        row_l = ahead, row_d = ahead_d;
        next_tile();
        if (t + 1 < n_iter) ahead = row_stat(r, true), ahead_d = row_stat(r, false);
      }
      if (!mbar_wait_warp(s_full, t & 1, abort_flag, p.status, kTimeoutTmemFull)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t sv[AB_COLS];
#pragma unroll
      for (int c = 0; c < AB_COLS / 32; ++c) tmem_ld_32x32(tmem_S + col + c * 32, reinterpret_cast<uint32_t(&)[32]>(sv[c * 32]));
      tmem_ld_wait();
      if (!OVER) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
      }
      // dP^T or dP: without OVER it is on its way while the exponentials are taken
      uint32_t dv[AB_COLS];
      auto load_dp = [&] {
        if (!mbar_wait_warp(dp_full, t & 1, abort_flag, p.status, kTimeoutTmemFull)) return false;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < AB_COLS / 32; ++c) tmem_ld_32x32(tmem_dP + col + c * 32, reinterpret_cast<uint32_t(&)[32]>(dv[c * 32]));
        return true;
      };
      if (!OVER && !load_dp()) {
        ok = false;
        break;
      }
      const float nl_row = scaled(row_l, true), nd_row = scaled(row_d, false);
      float2 pr[AB_COLS / 2];
      auto exponentials = [&](auto masks) {
#pragma unroll
        for (int i = 0; i < AB_COLS / 2; i += 2) {
          float4 n4 = make_float4(nl_row, nl_row, nl_row, nl_row);
          if (OVER) n4 = *reinterpret_cast<const float4*>(nl + 2 * i);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const float2 xs = __ffma2_rn(make_float2(__uint_as_float(sv[2 * (i + x)]), __uint_as_float(sv[2 * (i + x) + 1])), sc2,
                                         x ? make_float2(n4.z, n4.w) : make_float2(n4.x, n4.y));
            pr[i + x] = make_float2(exp2f(xs.x), exp2f(xs.y));
            // keys behind the query: rows above the column (OVER) or columns behind the row
            const int c = part * AB_COLS + 2 * (i + x);
            if (masks.value == kAll || (masks.value == kDiagonal && diag)) {
              if (OVER ? c < r : c > r) pr[i + x].x = 0.f;
              if (OVER ? c + 1 < r : c + 1 > r) pr[i + x].y = 0.f;
            }
          }
        }
      };
      // (beside the exponentials, which take longer, the masks cost nothing; a pass of their own behind them made short sequences 4 to 11 % slower)
      if constexpr (MASKS == kDiagonal) exponentials(Masks<kDiagonal>());
      else if (MASKS == kAll || diag) exponentials(Masks<kAll>());
      else exponentials(Masks<kNone>());
      if (!OVER) {
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(dp_free);
      }
      // P and dS in shared memory: chunk g of eight columns of this thread's row
      const int roff = part * 16384 + (r >> 3) * 1024 + (r & 7) * 128;
      auto put = [&](uint8_t* tile, int g, uint4 v) { *reinterpret_cast<uint4*>(tile + roff + ((g ^ (r & 7)) << 4)) = v; };
      uint32_t pk[VIA_SMEM ? 32 : 1];
      if (VIA_SMEM)
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] = pack_bf16x2(pr[i].x, pr[i].y);
      if (OVER) {   // (S of this iteration was written behind the product that read the P before it)
#pragma unroll
        for (int c = 0; c < 32; c += 16) {   // (half a row at a time: registers)
          uint32_t half[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) half[i] = pack_bf16x2(pr[c + i].x, pr[c + i].y);
          tmem_st_32x16(tmem_P + bf_col + c, half);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
        if (!load_dp()) {
          ok = false;
          break;
        }
        tmem_ld_wait();
      }
      uint32_t dk[32];
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float4 n4 = make_float4(nd_row, nd_row, nd_row, nd_row);
        if (OVER) n4 = *reinterpret_cast<const float4*>(nl + 128 + 2 * i);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float2 dd = __fmul2_rn(pr[i + x], __ffma2_rn(make_float2(__uint_as_float(dv[2 * (i + x)]), __uint_as_float(dv[2 * (i + x) + 1])), scale2,
                                                             x ? make_float2(n4.z, n4.w) : make_float2(n4.x, n4.y)));
          dk[i + x] = pack_bf16x2(dd.x, dd.y);
        }
      }
      // the products of the previous iteration must be done with P and dS before they are overwritten
      if (!OVER && !mbar_wait_warp(ds_free, (t & 1) ^ 1, abort_flag, p.status, kTimeoutTmemEmpty)) {
        ok = false;
        break;
      }
      if (VIA_SMEM) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          put(sP, g, make_uint4(pk[4 * g], pk[4 * g + 1], pk[4 * g + 2], pk[4 * g + 3]));
          put(sDS, g, make_uint4(dk[4 * g], dk[4 * g + 1], dk[4 * g + 2], dk[4 * g + 3]));
        }
        fence_proxy_async_smem();
      } else {
        tmem_st_32x32(tmem_dS + bf_col, dk);
        tmem_st_wait();
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    if (ok && mbar_wait_warp(acc_done, 0, abort_flag, p.status, kTimeoutTmemFull)) {
      tc_fence_after();
      const bool real = fixed * 128 + r < p.L;
      const long long tok = (long long)b * p.L + fixed * 128 + r;
      __nv_bfloat16* o1 = MODE == 0 ? p.dv + tok * p.ld_dkv + head * D : p.dq + tok * p.ld_dq + head * D;
      __nv_bfloat16* o2 = MODE == 0 ? p.dk + tok * p.ld_dkv + head * D : nullptr;
      // the AB_SPLIT threads of a row store D / AB_SPLIT columns each, 16 at a time
      constexpr int PIECES = D / 16 / AB_SPLIT;
#pragma unroll
      for (int c = part * PIECES; c < (part + 1) * PIECES; ++c) {
        uint32_t v[16];
        tmem_ld_32x16(tmem_A1 + lane_base + c * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 2; ++g)
          if (real) *reinterpret_cast<uint4*>(o1 + c * 16 + g * 8) =
              make_uint4(pack_bf16x2(__uint_as_float(v[8 * g]), __uint_as_float(v[8 * g + 1])), pack_bf16x2(__uint_as_float(v[8 * g + 2]), __uint_as_float(v[8 * g + 3])),
                         pack_bf16x2(__uint_as_float(v[8 * g + 4]), __uint_as_float(v[8 * g + 5])), pack_bf16x2(__uint_as_float(v[8 * g + 6]), __uint_as_float(v[8 * g + 7])));
        if (MODE == 0) {
          tmem_ld_32x16(tmem_A2 + lane_base + c * 16, v);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 2; ++g)
            if (real) *reinterpret_cast<uint4*>(o2 + c * 16 + g * 8) =
                make_uint4(pack_bf16x2(__uint_as_float(v[8 * g]), __uint_as_float(v[8 * g + 1])), pack_bf16x2(__uint_as_float(v[8 * g + 2]), __uint_as_float(v[8 * g + 3])),
                           pack_bf16x2(__uint_as_float(v[8 * g + 4]), __uint_as_float(v[8 * g + 5])), pack_bf16x2(__uint_as_float(v[8 * g + 6]), __uint_as_float(v[8 * g + 7])));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace ats

using namespace ats;

template <int D, int MODE, int FORM>
static int launch_attn_bwd(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                           const AttnBwdArgs& p, cudaStream_t s) {
  using SM = AttnBwdSmem<D, MODE, FORM>;
  cudaError_t ce = cudaFuncSetAttribute(attn_bwd_kernel<D, MODE, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL);
  if (ce != cudaSuccess) return int(ce);
  dim3 grid(MODE == 0 ? p.Hkv : p.Hq, p.B, (p.L + 127) / 128);
  attn_bwd_kernel<D, MODE, FORM><<<grid, AB_THREADS, SM::TOTAL, s>>>(mq, mk, mv, mdo, p);
  return int(cudaGetLastError());
}

// q/k/v as for ats_attn_fwd; out, dout: [B, L, Hq, D] contiguous; lse [B, Hq, L]; delta: fp32 scratch [B, Hq, L];
// dq: rows = tokens with pitch ld_dq, dk / dv with pitch ld_dkv (so all three can be slices of one packed gradient).
// prof: null, or 32 int64 that receive cycle totals of CTA (0,0,0) of each pass (diagnostics).
ATS_API int ats_attn_bwd(const void* q, long long ld_q, long long q_cols, int q_col0, const void* k, long long ld_k,
                         long long k_cols, int k_col0, const void* v, long long ld_v, long long v_cols, int v_col0,
                         const void* out, const void* dout, const float* lse, float* delta, void* dq, void* dk, void* dv,
                         long long ld_dq, long long ld_dkv, int B, int L, int Hq, int Hkv, int D, int* status, long long* prof, void* stream) {
  if ((D != 64 && D != 128) || L < 1 || Hq % Hkv || (q_col0 & 7) || (k_col0 & 7) || (v_col0 & 7) || (ld_dq & 7) || (ld_dkv & 7))
    return 1003;
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    cudaFree(0);
    ctx_bound = true;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CUtensorMap mq, mk, mv, mdo;
  int e;
  const unsigned long long n = L, od = (unsigned long long)Hq * D;
  if ((e = make_tmap_batched(&mq, q, q_cols, n, B, ld_q, n * ld_q, 128))) return e;
  if ((e = make_tmap_batched(&mk, k, k_cols, n, B, ld_k, n * ld_k, 128))) return e;
  if ((e = make_tmap_batched(&mv, v, v_cols, n, B, ld_v, n * ld_v, 128))) return e;
  if ((e = make_tmap_batched(&mdo, dout, od, n, B, od, n * od, 128))) return e;
  const long long delta_threads = (long long)B * L * Hq * (D / 8);
  attn_delta_kernel<<<unsigned((delta_threads + 255) / 256), 256, 0, s>>>(static_cast<const __nv_bfloat16*>(dout),
                                                                      static_cast<const __nv_bfloat16*>(out), delta, B, L, Hq, D);
  AttnBwdArgs p;
  p.B = B; p.L = L; p.Hq = Hq; p.Hkv = Hkv; p.D = D;
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.lse = lse; p.delta = delta;
  p.dq = static_cast<__nv_bfloat16*>(dq); p.dk = static_cast<__nv_bfloat16*>(dk); p.dv = static_cast<__nv_bfloat16*>(dv);
  p.ld_dq = ld_dq; p.ld_dkv = ld_dkv;
  p.scale = 1.f / sqrtf(float(D));
  p.scale_log2 = 1.4426950408889634f * p.scale;
  p.status = status;
  p.prof = prof;
  const bool one_pair = L <= 128 && Hq == Hkv, many = L > 8 * 128;
  if (D == 64) e = launch_attn_bwd<64, 0, 0>(mq, mk, mv, mdo, p, s);
  else if (one_pair) e = launch_attn_bwd<128, 0, 1>(mq, mk, mv, mdo, p, s);
  else e = launch_attn_bwd<128, 0, 0>(mq, mk, mv, mdo, p, s);
  if (e) return e;
  if (prof) p.prof = prof + 16;
  if (D == 64) return many ? launch_attn_bwd<64, 1, 1>(mq, mk, mv, mdo, p, s) : launch_attn_bwd<64, 1, 0>(mq, mk, mv, mdo, p, s);
  return many ? launch_attn_bwd<128, 1, 1>(mq, mk, mv, mdo, p, s) : launch_attn_bwd<128, 1, 0>(mq, mk, mv, mdo, p, s);
}
