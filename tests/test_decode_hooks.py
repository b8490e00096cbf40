"""What hangs on a module's call is seen by a captured decode step too: hooks, replaced modules, calibration."""
import pytest
import torch

from adaptivetrainingsystem_b200.config import ModelConfig
from adaptivetrainingsystem_b200.models import transformer as TR
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


def _model():
    torch.manual_seed(0)
    cfg = ModelConfig(vocab_size=512, hidden_size=256, num_layers=3, num_heads=4, num_kv_heads=2, intermediate_size=512, seq_length=64, tie_word_embeddings=False)
    return TR.DeepSeekTransformer(cfg).cuda().to(torch.bfloat16).eval()


def _steps(model, captured):
    """Logits of four decode steps behind a prompt, captured or one kernel at a time."""
    from adaptivetrainingsystem_b200.inference.engine import GenerationEngine
    ids = torch.randint(0, 512, (3, 12), generator=torch.Generator().manual_seed(1)).cuda()
    eng, cache = GenerationEngine(model), model.make_cache(3, 32)
    with torch.no_grad():
        eng.prefill(ids[:, :8], cache)
        dec = eng.graph_decoder(cache) if captured else None
        return torch.stack([(dec.step(ids[:, 8 + i]) if captured else eng.decode_step(ids[:, 8 + i], cache)).float() for i in range(4)])


class _Doubled(torch.nn.Module):
    """A feed-forward of the caller's own."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, h, residual=None):
        y, _ = self.inner(2 * h)
        return y + residual, None


def _halve(module, args, out):
    return (out[0] * 0.5, *out[1:]) if isinstance(out, tuple) else out * 0.5


def _plus_one(module, args):
    return (args[0] + 1, *args[1:])


# layer 1 stands between layers that fold their norms
@pytest.mark.gpu
@pytest.mark.parametrize("change", ["nothing", "hook on the feed-forward", "hook in front of the attention", "hook on the last norm", "feed-forward replaced", "forward replaced"])
def test_captured_step(change):
    from adaptivetrainingsystem_b200 import ops
    model = _model()
    plain = _steps(model, True)
    blk = model.layers[1]
    if change == "hook on the feed-forward":
        blk.ffn.register_forward_hook(_halve)
    elif change == "hook in front of the attention":
        blk.self_attn.register_forward_pre_hook(_plus_one)
    elif change == "hook on the last norm":
        model.norm.register_forward_hook(_halve)
    elif change == "feed-forward replaced":
        blk.ffn = _Doubled(blk.ffn)
    elif change == "forward replaced":
        inner = blk.ffn.forward
        blk.ffn.forward = lambda h, residual=None: inner(2 * h, residual)
    got, want = _steps(model, True), _steps(model, False)
    ops.check_status()
    # bf16 layers whose roundings differ: 2^-9 each in three layers of two sublayers, well below what any of the changes does
    assert float((got - want).norm() / want.norm()) < 2e-2
    if change != "nothing":
        assert float((got - plain).norm() / plain.norm()) > 0.1
