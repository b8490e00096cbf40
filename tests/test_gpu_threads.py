"""Decode kernels called from a thread that has not used the device before (a server's worker thread)."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["product", "swiglu", "attention"])
def test_first_call_of_a_thread(what):
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import gemm as G, serving
    g = torch.Generator(device="cuda").manual_seed(0)
    a, w = torch.randn(4, 256, generator=g, device="cuda").bfloat16(), torch.randn(512, 256, generator=g, device="cuda").bfloat16()
    cache, qkv = torch.randn(2, 4, 64, 2, 64, generator=g, device="cuda").bfloat16(), torch.randn(4, 1, 8 * 64, generator=g, device="cuda").bfloat16()
    out = torch.empty(4, 512, dtype=torch.bfloat16, device="cuda")   # (an allocation could select the device)
    run = {"product": lambda: G.gemm_nt(a, w, out=out), "swiglu": lambda: G.gemm_nt_swiglu(a, w, out=out[:, :256])}.get(what, lambda: serving.decode_attention(qkv, cache[0], cache[1], 3, 4, 2, 64))
    want = run().clone()
    torch.cuda.synchronize()
    got = []

    def body():
        try:
            got.append(run())
        except Exception as e:   # noqa: BLE001  (reported by the assertion below)
            got.append(e)
        torch.cuda.synchronize()
    t = threading.Thread(target=body)
    t.start()
    t.join()
    assert isinstance(got[0], torch.Tensor), got[0]
    assert torch.equal(got[0], want)
    ops.check_status()
