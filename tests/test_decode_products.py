"""Which products of a handful of rows run on the decode kernel and over how many CTAs (``ops/gemm.py``)."""
import pytest
import torch

from adaptivetrainingsystem_b200.ops import gemm as G


def _ok(T, N, K, pair=False):
    a, w = torch.empty(1, K).expand(T, K), torch.empty(1, K).expand(2 * N if pair else N, K)
    return G.skinny_ok(a, w, N) if pair else G.skinny_ok(a, w)


# sizes on both sides of each line, where the two kernels were measured further apart than their repetitions
@pytest.mark.parametrize("T,N,K,pair,ok", [
    (1, 128256, 64, False, True), (16, 8, 14336, False, True), (32, 32000, 256, False, True), (32, 128256, 384, False, False), (33, 32000, 2048, False, True),
    (64, 128256, 1024, False, False), (64, 2048, 2048, False, True), (80, 2048, 512, False, True), (96, 2048, 512, False, False), (128, 64, 256, False, False),
    (128, 1024, 8192, False, False), (65, 512, 14336, False, False), (128, 2048, 2048, False, True), (128, 4096, 14336, False, True), (128, 8192, 1024, False, False),
    (32, 28672, 256, True, True), (48, 28672, 512, True, False), (48, 1024, 256, True, True), (64, 256, 256, True, False), (64, 8192, 4096, True, True),
    (64, 14336, 1024, True, False), (65, 1024, 256, True, False), (128, 2816, 512, True, False), (128, 2816, 1024, True, True), (129, 256, 2048, False, False)])
def test_lines(T, N, K, pair, ok):
    assert _ok(T, N, K, pair) is ok


def test_slices_run_at_once():
    for T in (1, 64, 65, 128):
        for width in (64, 128):
            for tiles in range(1, 400):
                for K in (64, 512, 1024, 4096, 14336):
                    s = G.skinny_splits(T, tiles * width, K, width)
                    assert s in (1, 2, 3, 4, 8) and s <= max(1, K // 256)
                    assert s == 1 or s * tiles <= (296 if T <= 64 else 148)
                    assert s <= 2 or s * tiles <= (264 if T <= 64 else 132)
