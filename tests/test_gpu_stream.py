"""Products of a decode step on the streaming kernel (``csrc/gemv_bf16.cu``) against float64 products of the same bf16 operands."""
import pytest
import torch

from adaptivetrainingsystem_b200.ops import gemm as G

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _operands(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    return [torch.randn(M, K + 8, generator=g, device=DEV).bfloat16()[:, :K], (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()], g


def _near(got, want, mass, K, roundings=1):
    """fp32 sums (K ulp of the absolute sum) rounded to bf16 (2^-9 each, doubled)."""
    assert bool(((got.double() - want).abs() <= roundings * 2.0 ** -8 * want.abs() + (K + 8) * 2.0 ** -23 * mass).all())


# rows around the token tiles, one tile and the most of them, reductions of one step, of no whole ring, and the longest
@pytest.mark.parametrize("M,N,K", [(1, 16, 64), (7, 2368, 2048), (8, 48, 1088), (9, 2368, 1088), (16, 112, 8192), (3, 128, 14336)])
def test_store(M, N, K):
    (x, w), g = _operands(M, N, K)
    assert G.stream_fits(M, N, K)
    ref, mass = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    out = torch.full((M, N + 16), 7.0, device=DEV, dtype=torch.bfloat16)
    G.skinny(x, w, out[:, :N], G.SK_STORE)
    _near(out[:, :N], ref, mass, K)
    assert bool((out[:, N:] == 7.0).all())
    add = torch.randn(M, N + 2, generator=g, device=DEV).bfloat16()[:, :N]
    norm = (1 + 0.1 * torch.randn(N, generator=g, device=DEV)).bfloat16()
    y, rows = (torch.empty(M, N, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    parts = torch.empty(M, G.norm_parts(M, N, K), device=DEV)
    G.skinny(x, w, y, G.SK_STORE, add=add, next_norm=(norm, rows, parts))
    _near(y, ref + add.double(), mass + add.double().abs(), K)
    ss = (y.double() ** 2).view(M, -1, 16).sum(-1)
    assert torch.equal(rows, y * norm) and parts.shape == ss.shape and bool(((parts.double() - ss).abs() <= 16 * 2.0 ** -23 * ss).all())
    # the parts of a row divide the sums of the next product, here and on the decode kernel
    if N % 64 == 0:
        (_, w2), _ = _operands(M, 256, N)
        r = torch.rsqrt((y.double() ** 2).mean(-1, keepdim=True) + 1e-6)
        for splits in (None, 1):
            z = torch.empty(M, 256, device=DEV, dtype=torch.bfloat16)
            G.skinny(rows, w2, z, G.SK_STORE, scale=(parts, 1e-6), splits=splits)
            _near(z, r * (rows.double() @ w2.double().t()), r * (rows.double().abs() @ w2.double().abs().t()), N + 8)


@pytest.mark.parametrize("M,I,K", [(1, 16, 64), (8, 4736, 512), (9, 1408, 2048), (16, 48, 192)])
def test_swiglu(M, I, K):
    (x, w), _ = _operands(M, 2 * I, K)
    assert G.stream_fits(M, I, K, G.SK_SWIGLU)
    out = torch.empty(M, I, device=DEV, dtype=torch.bfloat16)
    G.skinny(x, w, out, G.SK_SWIGLU, n=I, up_offset=I)
    gate, up = (x.double() @ w.double().t()).chunk(2, -1)
    want = torch.nn.functional.silu(gate) * up
    # gate and up are rounded to bf16 first (2^-9 each, silu's slope is at most 1.1), the result once more
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * (2 * want.abs() + 1.1 * gate.abs() * up.abs()) + 1e-4).all())


@pytest.mark.parametrize("M,heads,d,K", [(1, 1, 32, 64), (8, 74, 64, 512), (9, 5, 128, 1088), (16, 40, 64, 2048), (4, 3, 96, 4096)])
def test_rotated_heads(M, heads, d, K):
    N = heads * d
    (x, w), g = _operands(M, N, K)
    assert G.stream_fits(M, N, K, G.SK_ROPE, d)
    cols = (heads + 1) // 2 * d
    cos, sin = (torch.rand(50, d // 2, generator=g, device=DEV) * 2 - 1 for _ in range(2))
    pos = torch.randint(0, 50, (M,), generator=g, device=DEV, dtype=torch.int32)
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    G.skinny(x, w, out, G.SK_ROPE, act_cols=cols, chain=(cos, None, 0.0, sin, None, 0.0), head_dim=d, pos=pos)
    ref = x.double() @ w.double().t()
    tol = 2.0 ** -8 * ref.abs() + (K + 8) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())
    (a, b), (ta, tb) = (t[:, :cols].view(M, -1, 2, d // 2).unbind(2) for t in (ref, tol))
    c, s = (t[pos.long()].double()[:, None] for t in (cos, sin))
    want, bound = torch.stack([a * c - b * s, a * s + b * c], 2), torch.stack([ta * c.abs() + tb * s.abs(), ta * s.abs() + tb * c.abs()], 2)
    assert bool(((out[:, :cols].double().view_as(want) - want).abs() <= 2.0 ** -8 * want.abs() + 1.01 * bound).all())
    assert bool(((out[:, cols:].double() - ref[:, cols:]).abs() <= tol[:, cols:]).all())


def test_forms_outside_the_lines_keep_the_decode_kernel():
    for M, N, K, mode, d in [(17, 2048, 2048, G.SK_STORE, 0), (1, 2056, 2048, G.SK_STORE, 0), (1, 2048, 2056, G.SK_STORE, 0), (1, 2384, 2048, G.SK_STORE, 0), (9, 64, 8256, G.SK_STORE, 0),
                             (1, 4752, 1024, G.SK_SWIGLU, 0), (1, 1024, 2112, G.SK_SWIGLU, 0), (1, 2560, 2048, G.SK_ROPE, 16), (1, 4800, 2048, G.SK_ROPE, 64), (1, 64, 64, G.SK_GELU, 0)]:
        assert not G.stream_fits(M, N, K, mode, d), (M, N, K, mode)
