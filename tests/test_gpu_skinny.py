"""Decode-sized products (``csrc/gemm_skinny.cu``) against float64 products of the same bf16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows around the accumulator widths, weights around the 128-row (64 for SwiGLU) tile, reductions around the 64-element block, every slice count
SHAPES = [(1, 8, 8), (1, 2560, 2048), (16, 136, 72), (17, 120, 264), (31, 2048, 5632), (33, 1000, 1024), (64, 128, 2048), (65, 4104, 512), (128, 264, 4096), (3, 32000, 2048)]


def _operands(T, N, K, seed=0, pitch=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(T, K + pitch, generator=g, device="cuda").bfloat16()[:, :K]
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    return a, w, a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()


def _check(out, ref, mass, K, rounding):
    """fp32 accumulation in any order: K ulp of the absolute products' sum; the stored value adds its own rounding, twice where an
    intermediate is rounded first."""
    bound = K * 2.0 ** -23 * mass + rounding * ref.abs() + 1e-30
    assert bool(((out.double() - ref).abs() <= bound).all()), float(((out.double() - ref).abs() / bound).max())


@pytest.mark.parametrize("T,N,K", SHAPES)
def test_products(T, N, K):
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import gemm as G
    a, w, ref, mass = _operands(T, N, K, pitch=8)
    _check(G.gemm_nt(a, w), ref, mass, K, 2.0 ** -8)
    _check(G.gemm_nt(a, w, out_fp32=True), ref, mass, K, 0)
    res = torch.randn(T, N, device="cuda").bfloat16()
    out = torch.empty(T, N + 24, device="cuda", dtype=torch.bfloat16)[:, 8:N + 8]
    G.gemm_nt(a, w, out=out, add=res, alpha=0.5)
    _check(out, 0.5 * ref + res.double(), mass + res.double().abs(), K, 2.0 ** -8)
    for splits in (1, 2, 3, 4, 8):
        if splits > (K + 63) // 64:
            continue
        part = torch.empty(splits, T, N, device="cuda")
        G.skinny(a, w, part, G.SK_PART, splits=splits)
        _check(part.double().sum(0), ref, mass, K, 0)
        one = torch.empty(T, N, device="cuda")
        G.skinny(a, w, one, G.SK_F32, splits=splits)
        _check(one, ref, mass, K, 0)
    ops.check_status()


@pytest.mark.parametrize("T,N,K", [(1, 5632, 2048), (16, 72, 200), (40, 64, 128), (64, 2816, 1024), (128, 200, 2048)])
def test_element_wise_steps(T, N, K):
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import dyt, gemm as G, postnorm
    a, w, ref, mass = _operands(T, 2 * N, K, seed=1)
    out = G.gemm_nt_swiglu(a, w)
    # gate and up are rounded to bf16 first; silu's slope is below 1.1
    g, u = (ref[:, :N], ref[:, N:])
    want = g * torch.sigmoid(g) * u
    slack = (2.0 ** -8 * g.abs() + K * 2.0 ** -23 * mass[:, :N]) * 1.1 * u.abs() + (2.0 ** -8 * u.abs() + K * 2.0 ** -23 * mass[:, N:]) * (g * torch.sigmoid(g)).abs()
    assert bool(((out.double() - want).abs() <= 1.1 * slack + 2.0 ** -8 * want.abs() + 1e-5).all())
    w, ref, mass = w[:N].contiguous(), ref[:, :N], mass[:, :N]
    tiny = 1e-5 + 1.2 * K * 2.0 ** -23 * mass     # fast exponentials (a few 1e-6 at these magnitudes); slopes below 1.2
    out = postnorm.linear_silu(a, w, N // 2 // 8 * 8)
    want = torch.cat([(z := ref[:, :N // 2 // 8 * 8]) * torch.sigmoid(z), ref[:, N // 2 // 8 * 8:]], 1)
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + tiny).all())
    bias = torch.randn(N, device="cuda")
    out = dyt.linear_gelu(a, w, bias)
    want = torch.nn.functional.gelu(ref + bias.double(), approximate="tanh")
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + tiny + 1e-5 * (ref.abs() + bias.abs().double())).all())
    x = torch.randn(T, N, device="cuda")
    v = [torch.randn(N, device="cuda") for _ in range(4)]
    x64 = x.double() + torch.tanh(0.7 * (ref + bias.double())) * v[0].double() + v[1].double()
    h = dyt.linear_residual(a, w, bias, x, dyt.DytChain(v[0], v[1], 0.7, v[2], v[3], 0.4))
    assert bool(((x.double() - x64).abs() <= (tiny + 1e-6) * (1 + v[0].abs().double())).all())
    want = torch.tanh(0.4 * x64) * v[2].double() + v[3].double()
    assert bool(((h.double() - want).abs() <= 2.0 ** -8 * want.abs() + (tiny + 1e-5) * (1 + v[0].abs().double()) * (1 + v[2].abs().double())).all())
    ops.check_status()


@pytest.mark.parametrize("T,n_q,n_kv,d,K", [(1, 32, 4, 64, 2048), (5, 2, 1, 128, 512), (64, 3, 1, 16, 136), (33, 8, 2, 32, 1024), (128, 4, 4, 64, 256), (7, 2, 1, 48, 256)])
def test_rotated_projection(T, n_q, n_kv, d, K):
    """Packed q / k / v with q and k rotated in the product's launch (head sizes that divide the tile) or in the fold's."""
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import serving
    a, w, ref, mass = _operands(T, (n_q + 2 * n_kv) * d, K, seed=2)
    a = a.contiguous()
    cos, sin = ops.rope_tables(300, d, device="cuda")
    pos = torch.randint(0, 300, (T,), device="cuda", dtype=torch.int32)
    out = serving.qkv_rope(a, w, cos, sin, pos, n_q, n_kv, d).double().view(T, -1, d)
    x, m = ref.view(T, -1, d), mass.view(T, -1, d)
    c, s = cos[pos.long()].double()[:, None], sin[pos.long()].double()[:, None]
    u, v = x.chunk(2, -1)
    turned = torch.cat([u * c - v * s, u * s + v * c], -1)
    turned[:, n_q + n_kv:] = x[:, n_q + n_kv:]
    # the product is rounded to bf16 before it turns, the result after
    size = torch.cat([u.abs() + v.abs()] * 2, -1)
    slack = torch.cat([sum(m.chunk(2, -1))] * 2, -1) * K * 2.0 ** -23 + 2.0 ** -8 * size + 2.0 ** -8 * turned.abs() + 1e-6
    assert bool(((out - turned).abs() <= slack).all())
    ops.check_status()
