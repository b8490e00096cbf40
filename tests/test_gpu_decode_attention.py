"""Decode attention (``decode_attn_kernel`` of ``csrc/inference.cu``) against float64 attention over the same bf16 rows."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _attend(q, k, v, scale, cap):
    s = torch.einsum("hd,nhd->hn", q, k) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    p = torch.softmax(s, -1)
    return torch.einsum("hn,nhd->hd", p, v), torch.einsum("hn,nhd->hd", p, v.abs())


def _check(out, ref, mass, cap):
    """Probabilities are rounded to bf16 before the second product and the output once more: 2^-8 of the weighted absolute values; the
    approximate exponential stays below 2^-9 of it, and the approximate tanh (2^-11) moves a capped score by up to cap * 2^-11."""
    bound = (1.5 * 2.0 ** -8 + cap * 2.0 ** -11) * mass + 2.0 ** -8 * ref.abs() + 1e-6
    assert bool(((out.double() - ref).abs() <= bound).all()), float(((out.double() - ref).abs() / bound).max())


# lengths around the units of 32 and 16 keys, the last row of the cache, every group size, one and several clusters per head
@pytest.mark.parametrize("B,hkv,rep,d,max_len,lengths", [
    (4, 4, 8, 64, 96, (0, 31, 32, 95)), (3, 2, 4, 128, 50, (15, 16, 49)), (2, 3, 1, 64, 33, (1, 32)), (2, 1, 2, 128, 1, (0, 0)),
    (1, 1, 8, 64, 5000, (4999,)), (2, 1, 4, 128, 3000, (2999, 17)), (70, 4, 2, 64, 1300, (700,)), (65, 8, 4, 128, 300, (255,))])
@pytest.mark.parametrize("cached", [False, True])
def test_decode_attention(B, hkv, rep, d, max_len, lengths, cached):
    from adaptivetrainingsystem_b200.ops import serving
    g = torch.Generator(device="cuda").manual_seed(B * max_len + d)
    hq = hkv * rep
    rows = torch.randn(2, B + 1, max_len, hkv, d, generator=g, device="cuda").bfloat16()
    lens = torch.tensor([lengths[i % len(lengths)] for i in range(B)], dtype=torch.int32, device="cuda")
    behind = torch.arange(max_len, device="cuda")[None] > lens[:, None]
    rows[:, :B][:, behind] = float("nan")   # what an earlier generation left behind the new token is never used
    k, v = rows[0, :B], rows[1, :B]
    qkv = torch.randn(B, 1, (hq + 2 * hkv) * d, generator=g, device="cuda").bfloat16()
    at = torch.arange(B, device="cuda")
    new_k, new_v = qkv[:, 0, hq * d:(hq + hkv) * d].view(B, hkv, d), qkv[:, 0, (hq + hkv) * d:].view(B, hkv, d)
    want_k, want_v = k.clone(), v.clone()
    if not cached:
        k[at, lens.long()] = float("nan")
        want_k[at, lens.long()], want_v[at, lens.long()] = new_k, new_v
    gate, cap, scale = None, 0.0, 1.0 / math.sqrt(d)
    if cached:
        gate, cap, scale = torch.randn(B, hq + 8, generator=g, device="cuda").bfloat16()[:, :hq], 15.0, 0.2
        out = torch.empty(B, hq * d + 16, dtype=torch.bfloat16, device="cuda")
        serving.decode_attention_cached(qkv[:, 0], k.view(B, max_len, -1), v.view(B, max_len, -1), lens, hq, hkv, d, scale, cap, gate, out)
        out = out[:, :hq * d]
    else:
        out = serving.decode_attention(qkv, k, v, lens, hq, hkv, d)[:, 0]
    assert torch.equal(k.view(torch.int16), want_k.view(torch.int16)) and torch.equal(v.view(torch.int16), want_v.view(torch.int16))
    for b in range(0, B, max(1, B // 4)):
        n = int(lens[b]) + 1
        ref, mass = _attend(qkv[b, 0, :hq * d].view(hq, d).double(), want_k[b, :n].double().repeat_interleave(rep, 1), want_v[b, :n].double().repeat_interleave(rep, 1), scale, cap)
        if gate is not None:
            f = torch.sigmoid(gate[b].double())[:, None]
            ref, mass = ref * f, mass * f
        _check(out[b].view(hq, d), ref, mass, cap)
