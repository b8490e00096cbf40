"""Scans of the delta rules: four and eight value columns per lane (``csrc/delta_rule.cu``, ``csrc/channel_delta.cu``) are the same sums; on the tensor-core
scans, which have no such forms, a sequence is the same alone and among others."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# sequences on either side of the line (192 CTAs of 64 columns); vdim 96 and 100 leave the last CTA partly empty, dim 72 its state rows
@pytest.mark.parametrize("dim,vdim,B,L,mma", [(128, 128, 13, 41, False), (72, 96, 13, 8, False), (128, 100, 13, 9, False), (128, 128, 13, 41, True), (72, 96, 13, 8, True)])
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("fresh", [False, True])
def test_batch_against_single_sequences(monkeypatch, channel, dim, vdim, B, L, mma, fresh):
    from adaptivetrainingsystem_b200.ops import delta as D
    monkeypatch.setattr(D, "scan_pays", lambda *_: mma)
    g = torch.Generator(device="cuda").manual_seed(dim + vdim + L)
    H, KH = 8, 4
    s = (D.ChannelDeltaShape if channel else D.DeltaShape)(heads=H, kv_heads=KH, dim=dim, vdim=vdim, taps=4, eps=1e-5)
    width = (s.channels + 7) // 8 * 8
    assert not mma or D.scan_on_tensor_cores(torch.empty(1, width, dtype=torch.bfloat16), s)
    mixed = torch.randn(B * L, width, generator=g, device="cuda").bfloat16()
    rlen = 0.05 + 0.05 * torch.rand(B * L, 2 * KH, generator=g, device="cuda")
    gb = torch.rand(B * L, 2 * H, generator=g, device="cuda") * 0.5 + 0.5
    start = torch.randn(B, H, dim, vdim, generator=g, device="cuda")
    a, rate, bias = torch.randn(B * L, H * dim, generator=g, device="cuda").bfloat16(), -torch.rand(H, generator=g, device="cuda"), torch.randn(H * dim, generator=g, device="cuda")

    def scan(rows, state):
        if channel:
            return D.channel_delta_scan(mixed[rows], rlen[rows], gb[rows], a[rows], rate, bias, state, s, L, fresh)
        return D.delta_scan(mixed[rows], rlen[rows], gb[rows], state, s, L, fresh)
    state = start.clone()
    out = scan(slice(0, B * L), state)       # 2 x 8 x 13 = 208 CTAs of 64 columns
    assert bool(torch.isfinite(out.float()).all()) and bool(torch.isfinite(state).all())
    for b in range(0, B, 4):
        one = start[b:b + 1].clone()
        rows = slice(b * L, (b + 1) * L)
        assert torch.equal(scan(rows, one), out[rows])
        assert torch.equal(one, state[b:b + 1])
