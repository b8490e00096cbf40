// Products of a decode step: at most 128 activation rows against a weight that is read once, out[t, n] = sum_k a[t, k] w[n, k], bf16 in,
// fp32 accumulation.
//
// Such a product is a stream of the weight: its floor is N K 2 bytes at the copy bandwidth (2 to 10 us for the projections of a
// 2048-wide decoder), so what counts is that as many SMs as possible stream, and that they start early.  The general GEMM puts the activations on the 128
// accumulator rows and tiles N by 256: qkv of a 2048-wide model is 10 tiles (40 CTAs with its four reduction slices), the gate / up product
// 44, so a third of the SMs streamed.  Here the operands are swapped: 128 weight rows are the rows of the tensor-core tile and the tokens its
// columns (16 to 128 of them, so one token costs 1/8 of the accumulator instead of a full one), and the reduction of a tile is cut over a
// cluster of up to eight CTAs, so that a product of up to 64 tokens has up to two CTAs for every SM (2,048 outputs: 16 tiles, 128 CTAs), beyond
// that one, each with all of its ring (72 to 90 KB; 128 KB beyond 64 tokens) in flight.
// The slices are summed through distributed shared memory in a fixed order (every CTA of the cluster owns a block of the tokens), and the
// element-wise step that follows the product (a rotation of the heads among them) is done there: no partial products in memory and no second
// launch.  Steps on whole rows (a norm) keep their fold kernels: kSkPart writes the slices.
//
// Measured (us, graph replay, weights larger than L2 in turn; general kernel with its separate fold before): 2560 x 2048 one row 14.4 -> 7.0,
// 64 rows 15.2 -> 9.8; 11264 x 2048 21.0 -> 11.9 / 21.4 -> 16.0; 2048 x 5632 17.1 -> 9.0 / 17.2 -> 12.2; 28672 x 4096 55 -> 40 / 47.6 -> 45.7.
// What is left is start-up (a launch of 1024 x 1024 takes 4.8 us) and, with 64 rows, the exchange of the slices (2 to 3 us).
//
// An RMSNorm between two products needs no launch either (skinny.cuh): the first product writes its rows times the norm's weight and their
// sums of squares per tile, the second one scales its sums.  With it and the residual read under the product, one decode step of eight
// 2048-wide layers: one sequence 331 -> 312 us, 64 sequences 626 -> 581 us.
//
// In a chain of launches (common.cuh) the first ring of weight tiles is requested before the kernel waits for its predecessor, if the caller says
// that the weight is not a result of the same step (w_ready).
#include "skinny.cuh"
#include "typed.cuh"

namespace ats {

int make_tmap_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, int elem_bytes, uint32_t box_cols, uint32_t box_rows);

namespace {

template <int V>
struct Int {
  static constexpr int value = V;
};

constexpr int SK_ROWS = 128;      // weight rows of a tile
constexpr int SK_BK = 64;         // reduction elements of a stage
constexpr int SK_THREADS = 192;   // TMA warp, MMA warp, four epilogue warps
constexpr int SK_MAX_SPLIT = 8;   // portable cluster size
constexpr int SK_TOKENS = 144;    // 128 and the padding of the owners' shares

__host__ __device__ constexpr int sk_stage_bytes(int nt) { return SK_ROWS * 128 + nt * 128; }
// Ring depth: two CTAs per SM up to 64 tokens (2 x (ring + reduction buffer) <= 227 KB), one beyond.
__host__ __device__ constexpr int sk_stages(int nt) { return nt == 16 ? 5 : nt == 32 ? 4 : nt == 64 ? 3 : 4; }
// Tokens that one CTA of a cluster sums: a multiple of four, so that they travel as 16-byte vectors.
__host__ __device__ constexpr int sk_per_owner(int t, int splits) { return ((t + splits - 1) / splits + 3) & ~3; }
// [slice][group of four tokens][weight row][4] of the owned tokens, so that a warp writes and reads 512 consecutive bytes: splits x per_owner <= nt + 8 for 1, 2, 3, 4 and 8 slices (32 for up to 16 tokens).
__host__ __device__ constexpr int sk_red_tokens(int nt) { return nt < 32 ? 32 : nt + 8; }
__host__ __device__ constexpr int sk_red_bytes(int nt) { return sk_red_tokens(nt) * SK_ROWS * 4; }
__host__ __device__ constexpr int sk_smem_bytes(int nt) { return 1024 + sk_stages(nt) * sk_stage_bytes(nt) + 256 + sk_red_bytes(nt); }

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, const uint32_t (&v)[16], int i) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]) : "memory");
}

// Four tokens of weight row `n` leave as bf16, two neighbouring rows in one word: even lanes write tokens 0 and 2, odd lanes 1 and 3 of the pair.
__device__ __forceinline__ void sk_store4(__nv_bfloat16* out, long long ldo, int T, int t, int n, const float (&v)[4], bool row_ok) {
  const int odd = threadIdx.x & 1;
#pragma unroll
  for (int e = 0; e < 4; e += 2) {
    const float give = odd ? v[e] : v[e + 1];
    const float got = __shfl_xor_sync(0xffffffffu, give, 1);
    const int tt = t + e + odd;
    if (row_ok && tt < T) *reinterpret_cast<uint32_t*>(out + (long long)tt * ldo + (n - odd)) = odd ? pack_bf16x2(got, v[e + 1]) : pack_bf16x2(v[e], got);
  }
}

__device__ __forceinline__ void sk_store4(const SkinnyArgs& p, int t, int n, const float (&v)[4], bool row_ok) {
  sk_store4(static_cast<__nv_bfloat16*>(p.out), p.ldo, p.T, t, n, v, row_ok);
}

// The element-wise steps that need no other row: one weight row n, four tokens at a time (the whole warp calls).
template <int MODE>
struct RowStep {
  static constexpr bool kDyt_ = MODE == kSkDyt;
  const SkinnyArgs& p;
  const int n;
  const bool row_ok;
  bool act = false;
  float bias = 0.f, w1 = 0.f, b1 = 0.f, w2 = 0.f, b2 = 0.f, next_w = 0.f;
  __device__ __forceinline__ RowStep(const SkinnyArgs& args, int row) : p(args), n(row), row_ok(row < args.N) {
    if (MODE == kSkSilu) act = n < p.act_cols;
    if (row_ok && (kDyt_ || MODE == kSkGelu) && p.bias) bias = p.bias[n];
    if (row_ok && kDyt_) w1 = p.w1[n], b1 = p.b1[n], w2 = p.w2[n], b2 = p.b2[n];
    if (row_ok && MODE == kSkStore && p.next_out) next_w = __bfloat162float(p.next_w[n]);
  }
  // Clamped, not guarded: guarded loads are waited for one by one (with one slice and 64 tokens that took 12 us).
  __device__ __forceinline__ void residual(int t, float (&r)[4]) const {
    const int nn = min(n, p.N - 1);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const long long tt = min(t + e, p.T - 1);
      r[e] = 0.f;
      if (MODE == kSkStore && p.add) r[e] = __bfloat162float(p.add[tt * p.ldadd + nn]);
      if (kDyt_) r[e] = p.x[tt * p.ldx + nn];
    }
  }
  // sq: where this warp leaves the sums of squares of the four tokens (kSkStore with next_out)
  __device__ __forceinline__ void finish(int t, float (&v)[4], float (&r)[4], float* sq) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool ok = row_ok && t + e < p.T;
      if (MODE == kSkF32) {
        if (ok) static_cast<float*>(p.out)[(long long)(t + e) * p.ldo + n] = v[e];
      } else if (kDyt_) {
        r[e] += tanh_fast(p.a1 * (v[e] + bias)) * w1 + b1;
        if (ok) p.x[(long long)(t + e) * p.ldx + n] = r[e];
        v[e] = tanh_fast(p.a2 * r[e]) * w2 + b2;
      } else if (MODE == kSkGelu) {
        v[e] = gelu_tanh_f<__nv_bfloat16>(v[e] + bias);
      } else if (MODE == kSkSilu) {
        v[e] = act ? silu_f(v[e]) : v[e];
      } else {
        v[e] += r[e];
      }
    }
    if (MODE != kSkF32) sk_store4(p, t, n, v, row_ok);
    if (MODE == kSkStore && p.next_out) {   // (the whole warp works on the same tokens)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float b = row_ok ? __bfloat162float(__float2bfloat16(v[e])) : 0.f;
        const float s = warp_sum(b * b);
        if ((threadIdx.x & 31) == 0) sq[e] = s;
        v[e] = b * next_w;
      }
      sk_store4(p.next_out, p.N, p.T, t, n, v, row_ok);
    }
  }
};

template <typename F>
__device__ __forceinline__ void by_mode(int mode, F&& f) {
  if (mode == kSkStore) f(Int<kSkStore>{});
  else if (mode == kSkF32) f(Int<kSkF32>{});
  else if (mode == kSkSilu) f(Int<kSkSilu>{});
  else if (mode == kSkGelu) f(Int<kSkGelu>{});
  else f(Int<kSkDyt>{});
}

// NT: token columns of the accumulator (tokens rounded up to 16, 32, 64 or 128).  grid (splits, tiles), cluster (splits, 1, 1) unless kSkPart.
template <int NT>
__global__ void __launch_bounds__(SK_THREADS)
skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const SkinnyArgs p, const int early) {
  constexpr int STAGES = sk_stages(NT), STAGE = sk_stage_bytes(NT);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);
  uint64_t* full = bars;             // [STAGES]
  uint64_t* empty = bars + STAGES;   // [STAGES]
  uint64_t* done = bars + 2 * STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* red = reinterpret_cast<float*>(smem + STAGES * STAGE + 256);
  // in the ring's memory once the product is done with it (shared memory of their own would keep small kernels of a chain off the SM)
  float* s_scale = reinterpret_cast<float*>(smem);                                                  // factor of a token's sums
  float(*s_sq)[SK_TOKENS] = reinterpret_cast<float(*)[SK_TOKENS]>(s_scale + SK_TOKENS);             // per epilogue warp and token: sum of squares of its 32 results

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = int(gridDim.x), split = int(blockIdx.x);   // a cluster spans the whole x dimension: its rank is the slice
  const bool swiglu = p.mode == kSkSwiglu;
  const int n0 = int(blockIdx.y) * (swiglu ? SK_ROWS / 2 : SK_ROWS);
  const int blocks = (p.K + SK_BK - 1) / SK_BK;
  const int kb0 = int((long long)blocks * split / S), kb1 = int((long long)blocks * (split + 1) / S);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_a);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, NT < 32 ? 32 : NT);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const bool reduce = S > 1 && p.mode != kSkPart;
  const int per = sk_per_owner(p.T, S);   // tokens of an owner
  // one slice and no partner row: the step is done on the accumulator's registers
  const bool direct = S == 1 && p.mode != kSkPart && p.mode != kSkSwiglu && p.mode != kSkRope;
  if (reduce) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // waited for before a peer's memory is written
  float ahead[8];

  auto sums_of_squares = [&](int from, int to) {   // of this tile's columns, in a fixed order
    for (int t = from + int(threadIdx.x) - 64; t < to; t += 128)
      p.next_parts[(long long)t * gridDim.y + blockIdx.y] = (s_sq[0][t] + s_sq[1][t]) + (s_sq[2][t] + s_sq[3][t]);
  };

  if (warp == 0) {
    if (lane == 0) {
      const int second = n0 + (swiglu ? p.up_offset : SK_ROWS / 2);
      auto weights = [&](int kb, int stage) {
        uint8_t* dst = smem + stage * STAGE;
        mbar_expect_tx(&full[stage], STAGE);
        tma_load_2d(dst, &map_w, &full[stage], kb * SK_BK, n0);
        tma_load_2d(dst + SK_ROWS / 2 * 128, &map_w, &full[stage], kb * SK_BK, second);
      };
      auto tokens = [&](int kb, int stage) { tma_load_2d(smem + stage * STAGE + SK_ROWS * 128, &map_a, &full[stage], kb * SK_BK, 0); };
      const int first = min(STAGES, kb1 - kb0);
      if (!early) asm volatile("griddepcontrol.wait;" ::: "memory");
      for (int i = 0; i < first; ++i) weights(kb0 + i, i);
      if (early) asm volatile("griddepcontrol.wait;" ::: "memory");
      for (int i = 0; i < first; ++i) tokens(kb0 + i, i);
      int stage = 0, phase = 0;
      for (int kb = kb0 + first; kb < kb1; ++kb) {
        if (!mbar_wait_bounded(&empty[stage], phase, abort_flag, p.status, kTimeoutEmpty)) break;
        weights(kb, stage);
        tokens(kb, stage);
        if (++stage == STAGES) stage = 0, phase ^= 1;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(SK_ROWS, NT, 1, 1, 0, 0);
      int stage = 0, phase = 0;
      bool ok = true;
      for (int kb = kb0; ok && kb < kb1; ++kb) {
        ok = mbar_wait_bounded(&full[stage], phase, abort_flag, p.status, kTimeoutFull);
        if (!ok) break;
        tc_fence_after();
        const uint64_t ad = make_smem_desc_sw128(smem_u32(smem + stage * STAGE), 0, 1024);
        const uint64_t bd = make_smem_desc_sw128(smem_u32(smem + stage * STAGE + SK_ROWS * 128), 0, 1024);
#pragma unroll
        for (int k = 0; k < SK_BK / 16; ++k) tc_mma_f16(tmem, desc_advance(ad, k * 32), desc_advance(bd, k * 32), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        tc_commit(&empty[stage]);
        if (++stage == STAGES) stage = 0, phase ^= 1;
      }
      if (ok) {
        tc_commit(done);
      } else {   // copies that were issued land before the CTA gives its shared memory back
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 10000000ull) {
        }
      }
    }
  } else {
    const int quad = warp & 3, row = quad * 32 + lane;   // tensor-memory lane = weight row of the tile
    asm volatile("griddepcontrol.wait;" ::: "memory");   // outputs may still be read, and residuals written, by the kernels before
    float factor = p.alpha;
    if (p.scale_parts && int(threadIdx.x) - 64 < p.T) {
      const float* parts = p.scale_parts + (long long)(int(threadIdx.x) - 64) * p.scale_n;
      float ss = 0.f;
      if ((p.scale_n & 3) == 0 && (reinterpret_cast<uintptr_t>(p.scale_parts) & 15) == 0) {  // (a streaming product leaves a part for every 16 columns)
#pragma unroll 8
        for (int i = 0; i < p.scale_n; i += 4) {
          const float4 v = *reinterpret_cast<const float4*>(parts + i);
          ss += v.x; ss += v.y; ss += v.z; ss += v.w;
        }
      } else {
#pragma unroll 8
        for (int i = 0; i < p.scale_n; ++i) ss += parts[i];
      }
      factor *= rsqrtf(ss * p.scale_inv + p.scale_eps);
    }
    if (reduce && p.mode == kSkStore && p.add) {   // the residual of the first eight owned tokens travels under the product
      const int nn = min(n0 + int(threadIdx.x) - 64, p.N - 1);
#pragma unroll
      for (int i = 0; i < 8; ++i) ahead[i] = __bfloat162float(p.add[(long long)min(split * per + i, p.T - 1) * p.ldadd + nn]);
    }
    const bool ok = mbar_wait_bounded(done, 0, abort_flag, p.status, kTimeoutTmemFull);
    tc_fence_after();
    __syncwarp();
    if (p.mode != kSkPart) s_scale[int(threadIdx.x) - 64] = factor;
    if (direct) asm volatile("bar.sync 1, 128;" ::: "memory");   // (the other paths meet at a barrier of the CTA before they read it)
    if (reduce) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t mine = smem_u32(red) + uint32_t(split * per * SK_ROWS + row * 4) * 4;
    auto chunk = [&](int c, uint32_t (&v)[16]) {
      tmem_ld_32x16(tmem + (uint32_t(quad * 32) << 16) + c * 16, v);
      tmem_ld_wait();
    };
    if (direct) {
      by_mode(p.mode, [&](auto mode_c) {
        const RowStep<decltype(mode_c)::value> step(p, n0 + row);
#pragma unroll 1
        for (int c = 0; ok && c * 16 < p.T; ++c) {
          uint32_t v[16];
          float r[4][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) step.residual(c * 16 + 4 * i, r[i]);
          chunk(c, v);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float f[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) f[e] = __uint_as_float(v[4 * i + e]) * s_scale[c * 16 + 4 * i + e];
            if (c * 16 + 4 * i < p.T) step.finish(c * 16 + 4 * i, f, r[i], &s_sq[warp - 2][c * 16 + 4 * i]);
          }
        }
      });
      if (p.next_out) {
        asm volatile("bar.sync 1, 128;" ::: "memory");
        sums_of_squares(0, p.T);
      }
    } else {
#pragma unroll 1
      for (int c = 0; ok && c * 16 < p.T; ++c) {
        uint32_t v[16];
        chunk(c, v);
        if (p.mode == kSkPart) {
          if (n0 + row < p.N) {
            float* dst = static_cast<float*>(p.out) + ((long long)split * p.T + c * 16) * p.N + n0 + row;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c * 16 + i < p.T) dst[(long long)i * p.N] = __uint_as_float(v[i]) * p.alpha;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const int t = c * 16 + i;
            if (t < p.T) {
              const int owner = t / per, q = (t - owner * per) >> 2;
              const uint32_t at = mine + uint32_t(q) * (SK_ROWS * 16);
              if (owner == split) *reinterpret_cast<uint4*>(red + (split * per + 4 * q) * SK_ROWS + row * 4) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
              else st_cluster_v4(mapa_shared(at, owner), v, i);
            }
          }
        }
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  if (reduce && warp < 2) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (p.mode != kSkPart && !direct) {
    if (reduce) cluster_sync_all();   // the slices of this CTA's tokens are in `red`
    else __syncthreads();
    if (warp >= 2) {
      const int i0 = int(threadIdx.x) - 64, t0 = split * per, groups = (max(0, min(per, p.T - t0)) + 3) >> 2;
      auto sum4 = [&](int row, int q, float (&v)[4]) {
        const float* src = red + (q * SK_ROWS + row) * 4;
        v[0] = v[1] = v[2] = v[3] = 0.f;
#pragma unroll 4
        for (int s = 0; s < S; ++s) {
          const float4 a = *reinterpret_cast<const float4*>(src + s * SK_ROWS * per);
          v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] *= s_scale[t0 + 4 * q + e];
      };
      if (swiglu) {
        const int col = i0 & 63;
        for (int q = i0 >> 6; q < groups; q += 2) {   // (a warp works on one q: the exchange of sk_store4 stays inside it)
          float g[4], u[4];
          sum4(col, q, g);
          sum4(col + 64, q, u);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // activation of the bf16-rounded values, as a separate pass over the pre-activations would have it
            g[e] = silu_f(__bfloat162float(__float2bfloat16(g[e]))) * __bfloat162float(__float2bfloat16(u[e]));
          }
          sk_store4(p, t0 + 4 * q, n0 + col, g, n0 + col < p.N);
        }
      } else if (p.mode == kSkRope) {   // pairs of rows half a head apart
        const int half = p.head_dim >> 1, r = i0 & 63, head = r / half, j = r - head * half, row = head * p.head_dim + j, n = n0 + row;
        const bool turn = n < p.act_cols;   // q and k columns turn, v columns do not
        for (int q = i0 >> 6; q < groups; q += 2) {
          float x[4], y[4];
          sum4(row, q, x);
          sum4(row + half, q, y);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = t0 + 4 * q + e;
            if (turn && t < p.T) {
              // rounded to bf16 first: the values that a separate rotation would read
              const float a = __bfloat162float(__float2bfloat16(x[e])), b = __bfloat162float(__float2bfloat16(y[e]));
              const long long at = (long long)p.pos[t] * half + j;
              const float cs = p.w1[at], sn = p.w2[at];
              x[e] = a * cs - b * sn;
              y[e] = a * sn + b * cs;
            }
          }
          sk_store4(p, t0 + 4 * q, n, x, n < p.N);
          sk_store4(p, t0 + 4 * q, n + half, y, n < p.N);
        }
      } else {
        const int n = n0 + i0;
        auto finish = [&](auto mode_c) {   // one loop per step: the memory accesses of two groups of tokens overlap
          const RowStep<decltype(mode_c)::value> step(p, n);
          const bool have = reduce && p.mode == kSkStore && p.add;
#pragma unroll 2
          for (int q = 0; q < groups; ++q) {
            float v[4], r[4];
            if (have && q < 2) {
#pragma unroll
              for (int e = 0; e < 4; ++e) r[e] = q ? ahead[4 + e] : ahead[e];
            } else {
              step.residual(t0 + 4 * q, r);
            }
            sum4(i0, q, v);
            step.finish(t0 + 4 * q, v, r, &s_sq[warp - 2][t0 + 4 * q]);
          }
        };
        by_mode(p.mode, finish);
        if (p.next_out) {
          asm volatile("bar.sync 1, 128;" ::: "memory");
          sums_of_squares(t0, min(p.T, t0 + 4 * groups));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, NT < 32 ? 32 : NT);
  }
}

template <int NT>
int sk_launch(const CUtensorMap& mw, const CUtensorMap& ma, const SkinnyArgs& p, int splits, int tiles, cudaStream_t stream) {
  if (cudaError_t ce = cudaFuncSetAttribute(skinny_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, sk_smem_bytes(NT))) return int(ce);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits, tiles);
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = sk_smem_bytes(NT);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (p.mode != kSkPart && splits > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = splits;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaError_t ce = cudaLaunchKernelEx(&cfg, skinny_kernel<NT>, mw, ma, p, int(p.w_ready && chained_launches()));
  return int(ce != cudaSuccess ? ce : cudaGetLastError());
}

}  // namespace
}  // namespace ats

using namespace ats;

// a [T, K] (row pitch lda), w [N, K] (or [2 N, K] with up_offset rows between gate and up for kSkSwiglu, row pitch ldw); `splits` reduction
// slices (kSkPart: out is [splits, T, N] fp32), or 0 for the streaming kernel.  Both operands 16-byte aligned with row pitches of a multiple of 8.
ATS_API int ats_gemm_skinny(const void* a, long long lda, const void* w, long long ldw, long long w_rows, const SkinnyArgs* args, int splits, void* stream) {
  SkinnyArgs p = *args;
  if (splits == 0) return stream_product(a, lda, w, ldw, w_rows, p, static_cast<cudaStream_t>(stream));
  const int blocks = (p.K + SK_BK - 1) / SK_BK;
  if (p.T < 1 || p.T > 128 || p.N < 1 || p.K < 8 || splits < 1 || splits > blocks || (splits > SK_MAX_SPLIT && p.mode != kSkPart)) return 1003;
  const int nt = p.T <= 16 ? 16 : p.T <= 32 ? 32 : p.T <= 64 ? 64 : 128;
  const int width = p.mode == kSkSwiglu ? SK_ROWS / 2 : SK_ROWS, tiles = (p.N + width - 1) / width;
  if (tiles > 65535 || (p.mode != kSkPart && splits * sk_per_owner(p.T, splits) > sk_red_tokens(nt))) return 1003;
  // pairs of neighbouring columns are written together
  if (p.mode != kSkPart && p.mode != kSkF32 && ((p.N & 1) || (reinterpret_cast<uintptr_t>(p.out) & 3) || (p.ldo & 1))) return 1003;
  if (p.mode == kSkRope && (p.head_dim < 4 || 128 % p.head_dim || p.N % p.head_dim || p.act_cols % p.head_dim || !p.pos || !p.w1 || !p.w2)) return 1003;
  if ((p.scale_parts && (p.mode == kSkPart || p.scale_n < 1)) || (p.next_out && (p.mode != kSkStore || !p.next_w || !p.next_parts || (p.N & 1)))) return 1003;
  CUtensorMap mw, ma;
  if (int e = make_tmap_2d(&mw, w, w_rows, p.K, ldw, 2, SK_BK, SK_ROWS / 2)) return e;
  if (int e = make_tmap_2d(&ma, a, p.T, p.K, lda, 2, SK_BK, nt)) return e;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (nt) {
    case 16: return sk_launch<16>(mw, ma, p, splits, tiles, s);
    case 32: return sk_launch<32>(mw, ma, p, splits, tiles, s);
    case 64: return sk_launch<64>(mw, ma, p, splits, tiles, s);
    default: return sk_launch<128>(mw, ma, p, splits, tiles, s);
  }
}
