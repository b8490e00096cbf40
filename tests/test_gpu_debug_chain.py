"""A failed check in the bounds-checking build keeps the order of a chain of launches (``common.cuh``).

Runs in a child process so that this library, not the release one, backs the package's operators."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

CHILD = textwrap.dedent('''
    import os, sys, torch
    sys.path.insert(0, os.environ["ATS_REPO"])
    from adaptivetrainingsystem_b200 import ops
    from adaptivetrainingsystem_b200.ops import _lib, gemm as G, serving
    assert _lib.DEBUG_BUILD
    g = torch.Generator(device="cuda").manual_seed(0)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    K = 131072   # eight CTAs, some 50 us: all of them have started long before the product is there
    w, norm, qkv, cache = r(128, K), r(128), r(3, 1, 12 * 64), r(2, 3, 64, 2, 64)
    lengths = torch.tensor([5, 64, 7], dtype=torch.int32, device="cuda")   # the second one is behind the cache: caught before it becomes an address
    for _ in range(5):
        a = r(64, K)
        want = ops.rms_norm(G.gemm_nt(a, w), norm, 1e-6)
        torch.cuda.synchronize()
        with G.chained_launches():
            y = G.gemm_nt(a, w)
            serving.decode_attention(qkv, cache[0], cache[1], lengths, 8, 2, 64)
            got = ops.rms_norm(y, norm, 1e-6)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        try:
            ops.check_status()
            raise SystemExit("the length was not caught")
        except ops.KernelError as e:
            assert "decode attention" in str(e)
    print("ORDER_OK")
''')


def test_order_behind_a_failed_check():
    from adaptivetrainingsystem_b200.ops import _lib
    if not os.path.exists(_lib.DEBUG_LIB):
        _lib.build_debug()
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], env=dict(os.environ, ATS_DEBUG_BUILD="1", ATS_REPO=repo), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "ORDER_OK" in r.stdout, (r.stdout + r.stderr)[-3000:]
