"""``gemm_nt`` with residuals and results that the kernels' epilogues cannot address: transposed, expanded, oddly pitched, of another type."""
import pytest
import torch

from adaptivetrainingsystem_b200.ops import gemm as G
from kernel_recorder import launches  # noqa: F401

FORMS = ["transposed", "column", "row", "pitch", "shifted", "fp32", "three dimensions"]


def _form(what, M, N, device, gen):
    def r(*shape):
        return torch.randn(*shape, generator=gen, device=device).bfloat16()
    return {"transposed": lambda: r(N, M).t(), "column": lambda: r(M, 1).expand(M, N), "row": lambda: r(1, N).expand(M, N), "pitch": lambda: r(M, N + 1)[:, :N],
            "shifted": lambda: r(M, N + 8)[:, 1:N + 1], "fp32": lambda: r(M, N).float(), "three dimensions": lambda: r(M, 1, N)}[what]()


@pytest.mark.parametrize("what", [f for f in FORMS if f != "row"])
def test_no_kernel_is_given_such_an_operand(launches, what):  # noqa: F811
    g = torch.Generator().manual_seed(0)
    a, w = torch.randn(4, 2048).bfloat16(), torch.randn(64, 2048).bfloat16()
    G.gemm_nt(a, w, add=_form(what, 4, 64, "cpu", g))
    if what != "column":
        G.gemm_nt(a, w, out=_form(what, 4, 64, "cpu", g))
    for x in launches:
        assert x.mode == G.SK_F32 and not x.add and x.ldo == 64


# one slice, several of them, the general kernel and its slices
@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (5, 256, 2048), (64, 136, 4096), (100, 8192, 2048), (300, 264, 512)])
@pytest.mark.parametrize("what", FORMS)
def test_against_float64(M, N, K, what):
    from adaptivetrainingsystem_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    ref, mass = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()

    def check(out, want):   # fp32 sums in any order, one rounding of the result
        bound = K * 2.0 ** -23 * (mass + want.abs()) + 2.0 ** -8 * want.abs() + 1e-30
        assert bool(((out.double().reshape(M, N) - want).abs() <= bound).all())
    add = _form(what, M, N, "cuda", g)
    want = ref + add.double().reshape(M, N)
    check(G.gemm_nt(a, w, add=add), want)
    if add.dtype == torch.bfloat16 and add.dim() == 2:
        check(ops.linear(a, w, residual=add), want)
    if what not in ("column", "row"):
        out = _form(what, M, N, "cuda", g)
        assert G.gemm_nt(a, w, out=out, add=add, alpha=0.5) is out
        check(out, 0.5 * ref + add.double().reshape(M, N))
    ops.check_status()
