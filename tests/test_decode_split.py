"""How decode attention is cut over CTAs (``decode_split`` of ``csrc/inference.cu``): partial results only where few pairs share long caches."""
import ctypes
import os

import pytest

from adaptivetrainingsystem_b200.ops import _lib


def _parts(B, hkv, d, tokens):
    if not os.path.exists(_lib.CUDA_LIB):
        pytest.skip("the kernel library has not been built")
    f = ctypes.CDLL(_lib.CUDA_LIB).ats_decode_attn_parts
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int] * 4
    return f(B, hkv, d, tokens)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("pairs", [1, 3, 8, 32, 37, 64, 128, 256, 1000, 65535])
def test_partial_results_stay_in_one_wave(pairs, d):
    for tokens in (1, 31, 500, 4000, 32000, 200000, 2000000000 // 65536):
        parts = _parts(pairs, 1, d, tokens)
        # above one they belong to clusters of eight, and all of them run at once
        assert parts >= 1 and (parts == 1 or 8 * pairs * parts <= 384)
        if pairs >= 256:
            assert parts == 1
