"""Over how many CTAs a decode product is cut (``ops/gemm.py``)."""
from adaptivetrainingsystem_b200.ops import gemm as G


def test_slices_run_at_once():
    for T in (1, 64, 65, 128):
        for width in (64, 128):
            for tiles in range(1, 400):
                for K in (64, 512, 1024, 4096, 14336):
                    s = G.skinny_splits(T, tiles * width, K, width)
                    assert s in (1, 2, 3, 4, 8) and s <= max(1, K // 256)
                    assert s == 1 or s * tiles <= (296 if T <= 64 else 148)
                    assert s <= 2 or s * tiles <= (264 if T <= 64 else 132)
