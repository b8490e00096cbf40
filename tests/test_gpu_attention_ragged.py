"""Causal attention of sequences whose length is no multiple of a tile (``csrc/attention_fwd2_tcgen05.cu``, ``csrc/attention_bwd_tcgen05.cu``)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# lengths around the 128-row tiles and the pairs of them, single rows, both head sizes, with and without groups
@pytest.mark.parametrize("B,L,hq,hkv,d", [(3, 1, 2, 2, 64), (2, 127, 4, 2, 128), (2, 129, 4, 1, 64), (3, 255, 4, 4, 64), (2, 257, 8, 2, 128), (3, 1000, 4, 2, 64), (1, 333, 4, 4, 128), (2, 128, 3, 3, 128), (2, 1, 2, 2, 128), (1, 128, 4, 2, 128), (1, 1024, 2, 1, 64), (1, 1025, 2, 2, 64),
                                         (1, 1024, 2, 2, 128), (1, 1025, 2, 1, 128)])
def test_ragged_lengths(B, L, hq, hkv, d):
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import attention_native as N
    g = torch.Generator(device="cuda").manual_seed(L)
    qkv = torch.randn(B, L, (hq + 2 * hkv) * d, generator=g, device="cuda").bfloat16()
    if B > 1:
        qkv[1] = float("nan")   # one sequence never reaches its neighbours
    qkv.requires_grad_()
    dout = torch.randn(B, L, hq, d, generator=g, device="cuda").bfloat16()
    out = N.flash_attention_packed(qkv, hq, hkv, d)
    out.backward(dout)
    ops.check_status()
    for b in range(0, B, 2):
        x = qkv.detach()[b:b + 1].double().requires_grad_()
        ref = ops.attention_reference(*(t.view(1, L, -1, d) for t in x.split([hq * d, hkv * d, hkv * d], -1)))
        ref.backward(dout[b:b + 1].double())
        # P, dS and the results are rounded to bf16 (2^-9 each); rows of gradients are sums of differences of nearly equal numbers, so
        # they are held against the largest row: a wrong row, or one of another sequence, differs by about its own norm
        for what, got, want, tol in (("out", out[b:b + 1].view(1, L, -1, d), ref.view(1, L, -1, d), 2e-2),
                                     ("grad", qkv.grad[b:b + 1].view(1, L, -1, d), x.grad.view(1, L, -1, d), 3e-2)):
            err, size = (got.double() - want).norm(dim=-1), want.norm(dim=-1)
            assert bool((err <= tol * (size + 0.3 * size.amax((1, 2), keepdim=True))).all()), (what, float((err / size.clamp(min=1e-3)).max()))
