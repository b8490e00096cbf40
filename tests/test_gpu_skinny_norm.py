"""An RMSNorm folded into the two decode products around it (``csrc/gemm_skinny.cu``) against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tokens around the accumulator widths and the owners' shares, widths around the 128-row tile, one slice and clusters of them
@pytest.mark.parametrize("T,N,K,splits", [(1, 2048, 2048, 8), (5, 1000, 512, 4), (16, 136, 264, 2), (17, 2048, 5632, 8), (33, 520, 1024, 3), (64, 2048, 2048, 8), (64, 384, 256, 1),
                                          (96, 1024, 2048, 4), (128, 8, 64, 1)])
def test_norm_between_products(T, N, K, splits):
    from adaptivetrainingsystem_b200.ops import gemm as G
    g = torch.Generator(device="cuda").manual_seed(T + N)
    a, res = (torch.randn(T, n, generator=g, device="cuda").bfloat16() for n in (K, N))
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    norm = (1 + 0.1 * torch.randn(N, generator=g, device="cuda")).bfloat16()
    x, plain = (torch.empty(T, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    rows, parts = torch.full((T, N), float("nan"), device="cuda", dtype=torch.bfloat16), torch.full((T, (N + 127) // 128), float("nan"), device="cuda")
    G.skinny(a, w, x, G.SK_STORE, add=res, splits=splits, next_norm=(norm, rows, parts))
    G.skinny(a, w, plain, G.SK_STORE, add=res, splits=splits)
    assert torch.equal(x, plain)   # the result itself does not change
    assert torch.equal(rows, x * norm)
    ss = torch.nn.functional.pad(x.double() ** 2, (0, -N % 128)).view(T, -1, 128).sum(-1)
    assert bool(((parts.double() - ss).abs() <= 128 * 2.0 ** -23 * ss).all())
    # the second product: fp32 sums of the rounded rows (K ulp of the absolute sums), one reciprocal root (2^-21), for bf16 results their rounding
    M, eps = 256, 1e-6
    w2 = (torch.randn(M, N, generator=g, device="cuda") * N ** -0.5).bfloat16()
    r = torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + eps)
    ref, mass = r * (rows.double() @ w2.double().t()), r * (rows.double().abs() @ w2.double().abs().t())
    for s in (1, 2, 4):
        if s > (N + 63) // 64:
            continue
        out = torch.empty(T, M, device="cuda")
        G.skinny(rows, w2, out, G.SK_F32, splits=s, scale=(parts, eps))
        assert bool(((out.double() - ref).abs() <= (N + 8) * 2.0 ** -23 * mass).all())
    act = torch.empty(T, M // 2, device="cuda", dtype=torch.bfloat16)
    G.skinny(rows, w2, act, G.SK_SWIGLU, n=M // 2, up_offset=M // 2, scale=(parts, eps))
    gate, up = ref.chunk(2, -1)
    want = torch.nn.functional.silu(gate) * up
    # gate and up are rounded to bf16 first (2^-9 each, silu's slope is at most 1.1), the result once more
    bound = 2.0 ** -8 * (2 * want.abs() + 1.1 * gate.abs() * up.abs()) + 1e-5 * (1 + mass.chunk(2, -1)[0] * mass.chunk(2, -1)[1])
    assert bool(((act.double() - want).abs() <= bound).all())
