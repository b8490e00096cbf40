"""Calibration records the rows of the products that a decode step fuses."""
import pytest
import torch

from adaptivetrainingsystem_b200.ops import int4, int8, serving
from kernel_recorder import launches  # noqa: F401


@pytest.mark.parametrize("what", [int4, int8])
def test_calibration_sees_every_product(launches, monkeypatch, what):  # noqa: F811
    x, gate_up, down, norm = torch.randn(2, 64).bfloat16(), torch.randn(256, 64).bfloat16(), torch.randn(64, 128).bfloat16(), torch.ones(64).bfloat16()
    what.observe(True)
    try:   # none of these calls ``record``: the caller's ordinary product does
        assert serving.mlp_norm(x, gate_up, down, x, norm, 1e-6) is None
        assert serving.out_proj_norm(torch.randn(2, 128).bfloat16(), down, x, norm, 1e-6) is None
    finally:
        what.observe(False)
    assert not launches
