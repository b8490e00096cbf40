"""The kernel library replaced by one that launches nothing and keeps the arguments of the decode products."""
import ctypes

import pytest
import torch

from adaptivetrainingsystem_b200.ops import _lib, gemm as G


class Recorder:
    """Stands in for the kernel library: every entry point returns 0; calls of ``ats_gemm_skinny`` are kept."""

    def __init__(self):
        self.args, self.known = [], {}

    def __getattr__(self, name):
        if name not in self.known:
            class Entry:
                restype = argtypes = None

                def __call__(_, *a):
                    if name == "ats_gemm_skinny":
                        self.args.append(G._Skinny.from_buffer_copy(a[5]._obj))
                    return 0
            self.known[name] = Entry()
        return self.known[name]


@pytest.fixture
def launches(monkeypatch):
    lib = Recorder()
    monkeypatch.setattr(_lib, "cuda_lib", lambda: lib)
    monkeypatch.setattr(G, "_configured", False)
    monkeypatch.setattr(_lib, "use_cuda_kernels", lambda t: True)
    monkeypatch.setattr(_lib, "status_tensor", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(_lib, "stream_ptr", lambda device=None: ctypes.c_void_p(0))
    return lib.args
