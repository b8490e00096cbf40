"""Which sequences run on the packed attention kernels (``ops.attention_packed_available``)."""
import pytest
import torch

from adaptivetrainingsystem_b200 import ops
from adaptivetrainingsystem_b200.ops import _lib, attn


@pytest.fixture(autouse=True)
def _pretend(monkeypatch):
    monkeypatch.setattr(_lib, "use_cuda_kernels", lambda t: True)
    monkeypatch.setattr(attn, "_native_available", lambda: True)


# sizes on both sides of each line, where the two were measured further apart than their repetitions; multiples of 128 always run on the packed kernels
@pytest.mark.parametrize("B,L,n_q,n_kv,grad,native", [
    (8, 300, 32, 4, True, True), (64, 40, 32, 4, True, True), (64, 40, 32, 4, False, False), (1, 33, 16, 4, False, True), (3, 1000, 16, 4, True, True),
    (8, 2000, 16, 4, True, True), (8, 2000, 16, 4, False, False), (1, 2000, 16, 4, True, True), (1, 8000, 16, 4, True, False), (1, 3000, 8, 8, False, True), (1, 2000, 32, 4, True, False), (2, 2000, 32, 4, True, False), (1, 2000, 16, 16, True, True),
    (1, 4000, 32, 4, True, False), (4, 4000, 16, 16, True, False), (1, 8000, 32, 8, False, False), (1, 8064, 32, 8, False, True), (1, 4096, 32, 4, True, True),
    (5, 31, 8, 8, True, False), (0, 300, 8, 8, True, False), (70000, 33, 1, 1, True, False)])
def test_lines(B, L, n_q, n_kv, grad, native):
    qkv = torch.empty(B, L, (n_q + 2 * n_kv) * 64, device="meta", requires_grad=grad)
    assert ops.attention_packed_available(qkv, 64, L, n_q, n_kv) is native


def test_unknown_heads():
    qkv = torch.empty(2, 1500, 24 * 64, device="meta", requires_grad=True)
    assert not ops.attention_packed_available(qkv, 64, 1500) and ops.attention_packed_available(qkv, 64, 1500, 8, 8)
    with torch.no_grad():
        assert ops.attention_packed_available(qkv[:, :1000].contiguous(), 64, 1000)
        assert not ops.attention_packed_available(qkv.reshape(30, 100, -1), 64, 100)
