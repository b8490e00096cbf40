// Products of a decode step of up to sixteen tokens with a bf16 weight, as a stream of the weight through warps.
//
// gemm_skinny.cu puts 128 weight rows on a tensor-core tile and cuts the reduction over a cluster: start-up, the exchange of the slices and the
// barriers of a cluster are 3.2 us of every launch, where the weight of a 2,048-wide projection is streamed in 1.3.  Here a CTA owns 16 weight rows
// (or two such tiles), its sixteen or eight warps split the reduction, and each keeps its share of the weight in flight in a ring of asynchronous
// copies, as the 4-bit kernel does (int4.cu): a warp-level MMA takes the 16 rows as they are stored and up to eight tokens as its columns.  With a CTA
// for every SM the whole weight of a projection is requested at once, in a captured step under the kernel before where that leaves an SM free; there is no
// cluster and no tensor memory to set up.  It is bound by one round trip to memory, the fold of the warps and the launch (1.4 us for 64 x 256).
//
// Us a launch in a chain, weights larger than L2 in turn, gemm_skinny.cu / here: one row 2,048 x 2,048 4.5 / 2.9, 2,048 x 5,632 8.0 / 5.9, rotated
// 2,560 x 2,048 5.2 / 3.7, pairs of 2,816 x 1,024 4.8 / 3.3; sixteen rows 5.0 / 3.8, 8.3 / 7.3, 5.6 / 4.6, 5.1 / 4.1.  Which products come here:
// stream_fits() in ops/gemm.py.  Warps and ring are the fastest of nine forms (a ring of four steps for up to eight tokens, 16 warps:
// 2,048 x 5,632 5.2, eight warps 7.3, rings of two steps 7.4).  Ring and sums are 200 KB for a plain tile (144 with more than eight tokens), 168 and 160 for heads, 88 and 112
// for gate and up tiles: one CTA per SM, two of the last.  So where a launch has a CTA on every SM the next one asks for its weight as SMs become free, and with up to 2,048 terms,
// two steps a warp, half of a plain ring is not used.  The last template number bounds the registers.
#include "skinny.cuh"
#include "stream_step.cuh"

namespace ats {
namespace {

// bytes one warp holds per stage: 16 rows of 64 weights for R tiles, 64 activations of 8 NT tokens
__host__ __device__ constexpr int bf16_stage_bytes(int R, int NT) { return R * 2048 + NT * 1024; }

// One step of a warp: 64 reduction indices of its tiles.  Quarter warps read 64 consecutive bytes of a row at a time: lane (g, t) has indices 32 q + 8 t .. + 7
// of rows g and g + 8, q = 0, 1, and the same ones of token g; a sum does not care which of its terms an MMA calls 2t, 2t + 1, 2t + 8, 2t + 9.
template <int MODE, int WARPS, int NT, int DEPTH, int MINB>
__global__ void __launch_bounds__(WARPS * 32, MINB)
gemv_bf16_kernel(const __nv_bfloat16* __restrict__ w, long long ldw, const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ add,
                 long long ld_add, __nv_bfloat16* __restrict__ out, long long ld_out, int M, int N, int K, int early, const StreamStep st) {
  constexpr int R = MODE == kStreamStore ? 1 : 2;
  if (!early) pdl_prologue();   // early: a chained launch whose weight no kernel in flight writes: its first stages are requested under the kernel before it
  else asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ float s_red[WARPS][R][8 * NT][16];  // [warp][tile][token][feature of the tile]
  __shared__ float s_scale[8 * NT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n_steps = K >> 6;
  int tile[R];
  const __nv_bfloat16* wrow[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    tile[r] = stream_tile<MODE>(st, N, r);
    wrow[r] = w + (long long)(tile[r] * 16 + g) * ldw + 8 * t;
  }
  float c[R][NT][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int n = 0; n < NT; ++n) c[r][n][0] = c[r][n][1] = c[r][n][2] = c[r][n][3] = 0.f;
  bool tok[NT];  // this lane supplies token g of token tile n
  const __nv_bfloat16* xrow[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    tok[n] = 8 * n + g < M;
    xrow[n] = x + (long long)(tok[n] ? 8 * n + g : 0) * ldx + 8 * t;
  }
  extern __shared__ __align__(16) unsigned char ring[];
  constexpr int STAGE = bf16_stage_bytes(R, NT);
  unsigned char* my_ring = ring + warp * DEPTH * STAGE + lane * 16;
  auto w_slot = [&](int d, int r, int i) { return my_ring + d * STAGE + r * 2048 + i * 512; };  // i = 2 (row half) + q
  auto x_slot = [&](int d, int n, int q) { return my_ring + d * STAGE + R * 2048 + n * 1024 + q * 512; };
  auto issue_w = [&](int d, int S) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) cp_async16(w_slot(d, r, i), wrow[r] + (i >> 1) * 8 * ldw + S * 64 + (i & 1) * 32);
  };
  auto issue_x = [&](int d, int S) {
#pragma unroll
    for (int n = 0; n < NT; ++n)  // lanes without a token get zeros
#pragma unroll
      for (int q = 0; q < 2; ++q) cp_async16_or_zero(x_slot(d, n, q), xrow[n] + S * 64 + q * 32, tok[n]);
  };
  auto compute = [&](int d) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint4 xv[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n) xv[n] = *reinterpret_cast<const uint4*>(x_slot(d, n, q));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint4 a = *reinterpret_cast<const uint4*>(w_slot(d, r, q)), b = *reinterpret_cast<const uint4*>(w_slot(d, r, 2 + q));
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          mma_16816(c[r][n], a.x, b.x, a.y, b.y, xv[n].x, xv[n].y);
          mma_16816(c[r][n], a.z, b.z, a.w, b.w, xv[n].z, xv[n].w);
        }
      }
    }
  };
  // group i of this lane's copies holds step warp + WARPS i; one group is committed per step, empty past the end (an early launch has the weights of
  // the whole ring in its first group)
  if (early) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d)
      if (warp + d * WARPS < n_steps) issue_w(d, warp + d * WARPS);
    asm volatile("griddepcontrol.wait;" ::: "memory");
  }
#pragma unroll
  for (int d = 0; d < DEPTH; ++d) {
    if (warp + d * WARPS < n_steps) {
      if (!early) issue_w(d, warp + d * WARPS);
      issue_x(d, warp + d * WARPS);
    }
    cp_async_commit();
  }
  stream_scales<WARPS, NT>(st, M, s_scale);  // (while the first copies travel)
  for (int S0 = warp; S0 < n_steps; S0 += WARPS * DEPTH) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      const int S = S0 + d * WARPS;
      if (S < n_steps) {  // the same for every lane of the warp
        cp_async_wait<DEPTH - 1>();  // all but the DEPTH - 1 youngest groups have landed: this step's is among them
        compute(d);
        const int Sn = S + WARPS * DEPTH;
        if (Sn < n_steps) issue_w(d, Sn), issue_x(d, Sn);  // (a lane refills the slots that it has just read itself)
        cp_async_commit();
      }
    }
  }
  cp_async_wait<0>();
  // accumulator of token tile n: c[0], c[1] = feature g, tokens 8 n + 2t and + 1; c[2], c[3] = feature g + 8
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      s_red[warp][r][8 * n + 2 * t][g] = c[r][n][0];
      s_red[warp][r][8 * n + 2 * t + 1][g] = c[r][n][1];
      s_red[warp][r][8 * n + 2 * t][g + 8] = c[r][n][2];
      s_red[warp][r][8 * n + 2 * t + 1][g + 8] = c[r][n][3];
    }
  __syncthreads();
  stream_finish<MODE, WARPS, NT, true>(st, s_red, s_scale, tile, add, ld_add, out, ld_out, M, N);
}

template <int MODE, int WARPS, int NT, int DEPTH, int MINB>
int launch_gemv(int ctas, const __nv_bfloat16* w, long long ldw, const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* add, long long ld_add, __nv_bfloat16* out,
                long long ld_out, int M, int N, int K, int early, const StreamStep& st, cudaStream_t s) {
  constexpr int kRing = WARPS * DEPTH * bf16_stage_bytes(MODE == kStreamStore ? 1 : 2, NT);
  auto kernel = gemv_bf16_kernel<MODE, WARPS, NT, DEPTH, MINB>;
  if (cudaError_t ce = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRing)) return int(ce);
  return int(launch_pdl(kernel, dim3(ctas), dim3(WARPS * 32), kRing, s, w, ldw, x, ldx, add, ld_add, out, ld_out, M, N, K, early, st));
}

}  // namespace

// Takes kSkStore (+ add), kSkSwiglu and kSkRope of up to 16 tokens, N a multiple of 16 (of 32, and of the heads, for kSkRope), K of 64.
int stream_product(const void* a, long long lda, const void* w, long long ldw, long long w_rows, const SkinnyArgs& p, cudaStream_t s) {
  const int mode = p.mode == kSkStore ? kStreamStore : p.mode == kSkSwiglu ? kStreamSwiGLU : p.mode == kSkRope ? kStreamRope : -1;
  const int M = p.T, K = p.K, N = mode == kStreamSwiGLU ? 2 * p.N : p.N;
  if (mode < 0 || M < 1 || M > 16 || N < 16 || (p.N & 15) || K < 64 || (K & 63) || (lda & 7) || (ldw & 7) || w_rows < N || p.alpha != 1.f ||
      (reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) || (mode == kStreamSwiGLU && (p.up_offset != p.N || p.add)) ||
      (mode == kStreamRope && (N & 31)))
    return 1003;
  StreamStep st = {};
  st.scale_parts = p.scale_parts; st.scale_n = p.scale_n; st.scale_inv = p.scale_inv; st.scale_eps = p.scale_eps;
  st.next_w = p.next_w; st.next_out = p.next_out; st.next_parts = p.next_parts;
  st.pos = p.pos; st.cos_t = p.w1; st.sin_t = p.w2; st.act_cols = p.act_cols; st.head_dim = p.head_dim;
  if (!stream_step_ok(st, mode, N, p.add != nullptr)) return 1003;
  if (mode != kStreamRope) st.head_dim = 32;
  const int early = p.w_ready && chained_launches(), tiles = N / 16, pairs = tiles / 2;
  auto go = [&](auto launch, int ctas) {
    return launch(ctas, static_cast<const __nv_bfloat16*>(w), ldw, static_cast<const __nv_bfloat16*>(a), lda, p.add, p.ldadd, static_cast<__nv_bfloat16*>(p.out), p.ldo, M, N,
                  K, early, st, s);
  };
  const bool two = M > 8;
  if (mode == kStreamSwiGLU) return two ? go(launch_gemv<kStreamSwiGLU, 8, 2, 2, 2>, pairs) : go(launch_gemv<kStreamSwiGLU, 8, 1, 2, 3>, pairs);
  if (mode == kStreamRope) return two ? go(launch_gemv<kStreamRope, 8, 2, 3, 2>, pairs) : go(launch_gemv<kStreamRope, 8, 1, 4, 2>, pairs);
  return two ? go(launch_gemv<kStreamStore, 16, 2, 2, 1>, tiles) : go(launch_gemv<kStreamStore, 16, 1, 4, 1>, tiles);
}

}  // namespace ats
