"""The entry point of the gathering product takes the epilogues that its kernel has and refuses the others before it looks at a pointer."""
import ctypes
import os

import pytest

STORE, ADD, F32, SWIGLU, SWIGLU_BWD, GELU, DYT, SILU = range(8)


def _call(epilogue, up_offset=0):
    from adaptivetrainingsystem_b200.ops import _lib
    if not os.path.exists(_lib.CUDA_LIB):
        pytest.skip("the CUDA library has not been built")
    f = ctypes.CDLL(_lib.CUDA_LIB).ats_gemm_bf16_gathered
    vp, ci, cll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    f.restype, f.argtypes = ci, [vp, cll, vp, vp, cll, vp, ci, ci, ci, vp, ci, vp, ci, vp, ci, vp, ci, ci, ci, ci, ci, ci, vp, vp]
    return f(None, 256, None, None, 512, None, 2, 0, 128, None, 1, None, 512, None, 0, None, 0, 256, 512, 256, epilogue, up_offset, None, None)


@pytest.mark.parametrize("epilogue", [F32, SWIGLU_BWD, GELU, DYT, SILU, -1, 8])
def test_other_epilogues_are_refused(epilogue):
    assert _call(epilogue) == 1004


def test_up_rows_start_at_whole_pieces():
    assert _call(SWIGLU, up_offset=4) == 1004
