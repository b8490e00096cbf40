"""Chained launches (``ops.gemm.chained_launches``): weights, packed words and cached keys fetched under the kernel before.  The kernels sum in fixed
orders, so every replay of a chain equals the same calls one after the other bit by bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gen(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def r(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()

    def weight(n, k):
        return torch.nn.Parameter(r(n, k, scale=k ** -0.5), requires_grad=False)
    return r, weight


def _compare(run, x, fresh, state=()):
    """``run()`` reads the buffer ``x``; it is captured as a chain and replayed for several contents of it.  ``state``: buffers that it writes."""
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import gemm as G
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph), G.chained_launches():
        out = run()
    for _ in range(4):
        x.copy_(fresh())
        before = [s.clone() for s in state]
        want = [t.clone() for t in run()] + [s.clone() for s in state]
        for s, b in zip(state, before):
            s.copy_(b)
        for _ in range(3):   # also right behind each other: the last kernels of one step and the first of the next
            graph.replay()
        torch.cuda.synchronize()
        for got, ref in zip([*out, *state], want):
            assert torch.equal(got.view(torch.int16), ref.view(torch.int16))
    ops.check_status()


@pytest.mark.parametrize("T,K,N", [(1, 2048, 512), (16, 512, 1000), (33, 1024, 264), (64, 2048, 2048), (128, 1024, 1024)])
def test_products(T, K, N):
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import dyt, gemm as G, postnorm, serving
    r, weight = _gen(T)
    d, x, norm_k, norm_n = 64, r(T, K), r(K), r(N)
    w_store, w_pair, w_fold, w_next, w_silu = weight(N, K), weight(2 * N, K), weight(N, K), weight(256, N), weight(N, K)
    w_rope, cos_sin, pos = weight(6 * d, K), ops.rope_tables(300, d, device="cuda"), torch.arange(T, dtype=torch.int32, device="cuda")
    post = postnorm.PostNorm(0.5, torch.rand(N, device="cuda"), 1e-6, N)

    def run():
        h = ops.rms_norm(x, norm_k, 1e-6)
        y = G.gemm_nt(h, w_store, add=h[:, :N].contiguous() if N <= K else None)
        rows, parts = torch.empty(T, N, dtype=x.dtype, device="cuda"), torch.empty(T, (N + 127) // 128, device="cuda")
        z = torch.empty_like(rows)
        G.skinny(h, w_store, z, G.SK_STORE, add=y, next_norm=(norm_n, rows, parts))
        scaled = torch.empty(T, 256, dtype=x.dtype, device="cuda")
        G.skinny(rows, w_next, scaled, G.SK_STORE, scale=(parts, 1e-6))
        pair = torch.empty_like(z)
        G.skinny(h, w_pair, pair, G.SK_SWIGLU, n=N, up_offset=N)
        res = z.float()
        folded = postnorm.linear_postnorm(h, w_fold, res, post)
        gelu = dyt.linear_gelu(folded[:, :N // 8 * 8].contiguous(), w_next, None) if N % 8 == 0 else folded
        return (y, z, scaled, pair, folded, gelu, postnorm.linear_silu(h, w_silu, N // 2 // 8 * 8), serving.qkv_rope(h, w_rope, *cos_sin, pos, 4, 1, d),
                G.gemm_nt(pair, w_next, out_fp32=True).bfloat16(), ops.rms_norm(pair, norm_n, 1e-6))
    _compare(run, x, lambda: r(T, K))


@pytest.mark.parametrize("T", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(64, 256), (2560, 2048), (2048, 5632)])
def test_4_bit_products(T, N, K):
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import int4
    r, weight = _gen(T)
    x, norm_k, norm_n = r(T, K), r(K), r(N)

    def packed(n, k):
        q, scale, zero = int4.quantize_rtn(weight(n, k), 128)
        return int4.pack(q), int4.pack_meta(scale, zero)
    first, pair = packed(N, K), packed(2 * N, K)

    def run():
        h = ops.rms_norm(x, norm_k, 1e-6)
        y = int4.gemv(h, *first, 128, add=h[:, :N].contiguous() if N <= K else None)
        return y, int4.gemv(h, *pair, 128, swiglu=True), ops.rms_norm(y, norm_n, 1e-6)
    _compare(run, x, lambda: r(T, K))


# lengths on either side of the units of 32 (64 dimensions) and 16 keys, the first and the last row of the cache, one and several clusters a head
@pytest.mark.parametrize("hkv,rep,d,max_len,lengths", [(2, 4, 64, 96, (0, 31, 32, 33, 63, 64, 95)), (1, 8, 128, 50, (15, 16, 17, 49)), (1, 1, 64, 9000, (8000, 8191, 8192)), (4, 2, 128, 700, (255, 256, 699))])
def test_attention_that_appends(hkv, rep, d, max_len, lengths):
    from adaptivetrainingsystem_b200.ops import gemm as G, serving
    r, weight = _gen(max_len)
    B, K, hq = len(lengths), 256, hkv * rep
    x, w_qkv, w_o = r(B, K), weight((hq + 2 * hkv) * d, K), weight(K, hq * d)
    cache, lens = r(2, B, max_len, hkv, d), torch.tensor(lengths, dtype=torch.int32, device="cuda")

    def run():
        a = serving.decode_attention(G.gemm_nt(x, w_qkv).view(B, 1, -1), cache[0], cache[1], lens, hq, hkv, d)
        return a, G.gemm_nt(a[:, 0], w_o)
    _compare(run, x, lambda: r(B, K), [cache])


@pytest.mark.parametrize("G_,rep,d,max_len,lengths", [(2, 4, 64, 96, (0, 31, 32, 33, 63, 64, 95)), (1, 8, 128, 50, (15, 16, 17, 49)), (1, 1, 64, 9000, (8000, 8191, 8192)), (4, 2, 128, 700, (255, 256, 699))])
def test_attention_behind_the_append(G_, rep, d, max_len, lengths):
    """The row of the new token is written by the kernel right in front, and a second layer reads the same cache."""
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import gemm as G, gqa
    r, weight = _gen(max_len)
    B, K, H = len(lengths), 256, G_ * rep
    own = gqa.GqaShape(heads=H, kv_heads=G_, dim=d, vdim=d, rot=32, scale=0.2, cap=15.0, eps=1e-6)
    shared = gqa.GqaShape(heads=H, kv_heads=G_, dim=d, vdim=d, rot=32, scale=0.2, cap=15.0, eps=1e-6, own_kv=False)
    x, w_own, w_shared, w_o = r(B, K), weight(own.proj_width, K), weight(shared.proj_width, K), weight(K, own.o_pad)
    q_w, k_w = (torch.rand(n * d, device="cuda") + 0.5 for n in (H, G_))
    cos, sin = ops.rope_tables(max_len + 1, 32, device="cuda")
    cache, lens = r(2, B, max_len, G_ * d), torch.tensor(lengths, dtype=torch.int32, device="cuda")
    assert gqa.decode_tc_ok(torch.empty(B, own.q_pad, dtype=torch.bfloat16, device="cuda"), own, cache[0], cache[1])

    def run():
        outs = []
        h = x
        for s, w in ((own, w_own), (shared, w_shared)):
            proj = G.gemm_nt(h, w).view(B, 1, -1)
            q = gqa.gqa_prepare(proj, s, q_w, k_w if s.own_kv else None, cos, sin, cache[0], cache[1], lengths=lens)
            a = gqa.gqa_decode(q, cache[0], cache[1], proj[:, 0, s.g_col:], s, lens)
            h = G.gemm_nt(a, w_o)
            outs += [a, h]
        return tuple(outs)
    _compare(run, x, lambda: r(B, K), [cache])
