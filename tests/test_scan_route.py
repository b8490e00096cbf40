"""Which portions of the delta rules run on the tensor cores: the lines of the rule, and that batches play no part in it."""
import inspect

import pytest

from adaptivetrainingsystem_b200.ops import delta as D


@pytest.mark.parametrize("channel,dim,vdim,last_on_fmas", [(False, 128, 128, 40), (False, 72, 16, 40), (False, 64, 64, 8), (False, 16, 256, 8), (True, 128, 128, 64), (True, 96, 64, 64),
                                                          (True, 128, 56, None), (True, 64, 64, 8), (True, 40, 128, 8), (True, 32, 128, 24), (True, 64, 56, 24)])
def test_lines(channel, dim, vdim, last_on_fmas):
    s = (D.ChannelDeltaShape(heads=4, kv_heads=2, dim=dim, vdim=vdim, taps=4, eps=1e-5, decay_rank=8, gate_rank=8) if channel
         else D.DeltaShape(heads=4, kv_heads=2, dim=dim, vdim=vdim, taps=4, eps=1e-5))
    assert list(inspect.signature(D.scan_pays).parameters) == ["s", "L"]
    for L in (1, 8, 9, 24, 25, 40, 41, 64, 65, 4096):
        assert D.scan_pays(s, L) == (last_on_fmas is not None and L > last_on_fmas)
