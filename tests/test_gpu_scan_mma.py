"""Delta scans on the tensor cores (``csrc/delta_rule_mma.cu``, ``csrc/channel_delta_mma.cu``) against the recurrence in 64 bits and the scans in fp32 FMAs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def all_lengths_on_tensor_cores(monkeypatch):
    from adaptivetrainingsystem_b200.ops import delta as D
    monkeypatch.setattr(D, "scan_pays", lambda *_: True)


def _inputs(channel, B, L, H, KH, dim, vdim, shift, seed=None):
    from adaptivetrainingsystem_b200.ops import delta as D
    g = torch.Generator(device="cuda").manual_seed(B + L + H + dim + vdim if seed is None else seed)

    def r(*shape):
        return torch.randn(*shape, generator=g, device="cuda")
    if channel:
        s = D.ChannelDeltaShape(heads=H, kv_heads=KH, dim=dim, vdim=vdim, taps=4, eps=1e-5, decay_rank=8, gate_rank=8)
    else:
        s = D.DeltaShape(heads=H, kv_heads=KH, dim=dim, vdim=vdim, taps=4, eps=1e-5)
    proj, conv, tail = r(B, L, s.proj_width).bfloat16(), r(s.taps, s.channels) * 0.5, r(B, 3, s.channels).bfloat16()
    rate = -torch.exp(r(H) * 0.5)
    start = r(2 * B, H, dim, vdim)[::2]      # sequences that do not lie side by side
    if channel:
        mixed, rlen, gb = D.delta_prep(proj, s, conv, None, None, tail)
        a, bias = r(B * L, H * dim).bfloat16(), r(H * dim) * 0.5 + shift
        decay = torch.exp(rate.double()[:, None] * torch.nn.functional.softplus(a.double() + bias.double()).view(-1, H, dim)).view(B, L, H, dim)

        def scan(state, fresh):
            return D.channel_delta_scan(mixed, rlen, gb, a, rate, bias, state, s, L, fresh)
    else:
        mixed, rlen, gb = D.delta_prep(proj, s, conv, rate, r(H) * 0.5 + shift, tail)
        decay = gb.double()[:, :H].view(B, L, H, 1)

        def scan(state, fresh):
            return D.delta_scan(mixed, rlen, gb, state, s, L, fresh)
    return s, mixed, rlen, gb, decay, start, scan


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def _exact(s, mixed, rlen, gb, decay, start, L, fresh):
    B, H, KH, dim = start.shape[0], s.heads, s.kv_heads, s.dim
    m, rl = mixed.double(), rlen.double()
    q = (m[:, :KH * dim].view(B, L, KH, dim) * rl[:, :KH].view(B, L, KH, 1)).repeat_interleave(H // KH, 2)
    k = (m[:, KH * dim:2 * KH * dim].view(B, L, KH, dim) * rl[:, KH:].view(B, L, KH, 1)).repeat_interleave(H // KH, 2)
    v, beta = m[:, 2 * KH * dim:s.channels].view(B, L, H, s.vdim), gb.double()[:, H:].view(B, L, H, 1)
    S, out = (torch.zeros_like(start) if fresh else start).double(), []
    for t in range(L):
        S = S * decay[:, t, :, :, None]
        u = beta[:, t] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", S, k[:, t]))
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        out.append(torch.einsum("bhdv,bhd->bhv", S, q[:, t]))
    return torch.stack(out, 1).view(B * L, -1), S


# lengths around the groups of 16 tokens and their halves; state rows and columns around the tiles of 64, 128 and 16; one to three heads a key head
@pytest.mark.parametrize("B,L,H,KH,dim,vdim,slow", [(1, 1, 2, 2, 128, 128, False), (2, 8, 3, 1, 8, 8, False), (2, 15, 4, 2, 64, 96, True), (1, 16, 2, 1, 72, 40, False),
                                                    (3, 17, 3, 3, 128, 64, False), (1, 25, 6, 2, 120, 16, True), (2, 331, 4, 2, 128, 128, True)])
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("fresh", [False, True])
def test_against_recurrence_and_fma_scan(monkeypatch, channel, B, L, H, KH, dim, vdim, slow, fresh):
    from adaptivetrainingsystem_b200.ops import delta as D
    s, mixed, rlen, gb, decay, start, scan = _inputs(channel, B, L, H, KH, dim, vdim, -6.0 if slow else -2.0)
    assert D.scan_on_tensor_cores(mixed, s)
    state = start.clone()
    out = scan(state, fresh)
    want, S = _exact(s, mixed, rlen, gb, decay, start, L, fresh)
    monkeypatch.setattr(D, "scan_on_tensor_cores", lambda *_: False)
    fma_state = start.clone()
    fma_out = scan(fma_state, fresh)

    # Read-outs carry the rounding to bf16 (2^-9 an element at most).  States: 32-bit sums; with a decay per row the error of the fast exponential of
    # each token's decay (a few 1e-7) adds up over the tokens that a state remembers.  Neither is further off than the FMA scan by more than
    # rounding errors of a single draw differ from one order of sums to another; the test below compares their averages.
    assert _rel(out, want) < 2.0 ** -8
    assert _rel(state, S) < (4e-6 if channel else 6e-7)
    assert _rel(state, S) < 1.25 * _rel(fma_state, S) + 5e-9 and _rel(out, want) < _rel(fma_out, want) + 1e-5


# From slow decays to those that forget a token at once, where a state is no further from 64 bits than a few of its own roundings: on average over draws
# the scan is as close as the FMA scan (0.6 to 1.0 of its error; the mean of eight draws is good to 0.03).
@pytest.mark.parametrize("shift", [-6.0, -2.0, 0.0, 2.0, 5.0])
@pytest.mark.parametrize("L,dim", [(8, 64), (32, 64), (331, 128)])
@pytest.mark.parametrize("channel", [False, True])
def test_no_further_from_64_bits_than_the_fma_scan(monkeypatch, channel, L, dim, shift):
    from adaptivetrainingsystem_b200.ops import delta as D
    error = {True: 0.0, False: 0.0}
    for seed in range(8):
        s, mixed, rlen, gb, decay, start, scan = _inputs(channel, 4, L, 8, 4, dim, dim, shift, seed)
        _, S = _exact(s, mixed, rlen, gb, decay, start, L, False)
        for mma in error:
            with monkeypatch.context() as m:
                if not mma:
                    m.setattr(D, "scan_on_tensor_cores", lambda *_: False)
                state = start.clone()
                scan(state, False)
            error[mma] += _rel(state, S) / 8
    assert error[True] < 1.03 * error[False], error


# A value that is not finite reaches its own token and the later ones, as in the recurrence: in the first and the second eight tokens of a group, in a later
# group, in the values, keys, queries, decays (the channel-wise rule makes its own) and step sizes, and in the state at the start.
@pytest.mark.parametrize("channel,where", [(c, w) for c in (False, True) for w in ("v", "k", "q", "decay", "beta", "state") if not (c and w == "decay")])
@pytest.mark.parametrize("token,bad", [(5, float("nan")), (13, float("inf")), (27, float("-inf"))])
def test_values_that_are_not_finite_stay_behind_the_tokens_before_them(channel, where, token, bad):
    B, L, H, KH, dim, vdim = 2, 40, 4, 2, 64, 80
    if where in ("decay", "beta"):
        bad = float("nan")
    s, mixed, rlen, gb, decay, start, scan = _inputs(channel, B, L, H, KH, dim, vdim, -2.0)
    clean = scan(start.clone(), False)
    row = L + token                       # of the second sequence
    if where == "v":
        mixed[row, 2 * KH * dim + vdim + 3] = bad
    elif where in "kq":
        mixed[row, (KH * dim if where == "k" else 0) + dim + 7] = bad
    elif where == "decay":
        gb[row, 2] = bad
        decay = gb.double()[:, :H].view(B, L, H, 1)
    elif where == "beta":
        gb[row, H + 2] = bad
    else:
        start = start.clone()
        start[1, 2, 9, 4] = bad
    state = start.clone()
    out = scan(state, False)
    want, S = _exact(s, mixed, rlen, gb, decay, start, L, False)
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(out), finite) and torch.equal(torch.isfinite(state), torch.isfinite(S))
    assert not bool(finite.all()) and torch.equal(out[finite], clean[finite])


# Rows that do not start at 16-byte pieces (a slice of a wider matrix, an odd pitch) are copied to some that do: on both kinds of scan.
@pytest.mark.parametrize("channel", [False, True])
@pytest.mark.parametrize("dim,vdim", [(64, 48), (40, 20), (36, 20)])
@pytest.mark.parametrize("offset,pad", [(1, 8), (2, 7), (0, 5), (4, 4)])
def test_rows_at_any_address(channel, dim, vdim, offset, pad):
    from adaptivetrainingsystem_b200.ops import delta as D
    B, L, H, KH = 2, 21, 4, 2
    s = (D.ChannelDeltaShape(heads=H, kv_heads=KH, dim=dim, vdim=vdim, taps=4, eps=1e-5, decay_rank=8, gate_rank=8) if channel
         else D.DeltaShape(heads=H, kv_heads=KH, dim=dim, vdim=vdim, taps=4, eps=1e-5))
    g = torch.Generator(device="cuda").manual_seed(dim + offset)
    mixed = torch.randn(B * L, (s.channels + 7) // 8 * 8, generator=g, device="cuda").bfloat16()
    a = torch.randn(B * L, H * dim, generator=g, device="cuda").bfloat16()
    rlen, gb = 0.05 + 0.05 * torch.rand(B * L, 2 * KH, generator=g, device="cuda"), torch.rand(B * L, 2 * H, generator=g, device="cuda")
    rate, bias = -torch.rand(H, generator=g, device="cuda"), torch.randn(H * dim, generator=g, device="cuda")

    def elsewhere(t):
        wide = torch.zeros(t.shape[0], offset + t.shape[1] + pad, dtype=t.dtype, device="cuda")
        return wide[:, offset:offset + t.shape[1]].copy_(t)

    def scan(m, x):
        state = torch.ones(B, H, dim, vdim, device="cuda")
        return (D.channel_delta_scan(m, rlen, gb, x, rate, bias, state, s, L, False) if channel else D.delta_scan(m, rlen, gb, state, s, L, False)), state
    out, state = scan(mixed, a)
    for m, x in ((elsewhere(mixed), a), (mixed, elsewhere(a)), (elsewhere(mixed), elsewhere(a))):
        o, st = scan(m, x)
        assert torch.equal(o, out) and torch.equal(st, state)
