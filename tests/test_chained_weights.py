"""Which products of a chained decode step may fetch their weight under the kernel before them: those whose weight no kernel of the step writes."""
import pytest
import torch

from adaptivetrainingsystem_b200.ops import gemm as G, int4
from kernel_recorder import launches  # noqa: F401


def _weight(n=256, k=128):
    return torch.nn.Parameter(torch.randn(n, k).bfloat16(), requires_grad=False)


def test_parameters_are_ready(launches):
    a, w = torch.randn(4, 128).bfloat16(), _weight()
    G.gemm_nt(a, w)
    G.gemm_nt_swiglu(a, w)
    G.skinny_partials(a, w)
    assert [x.w_ready for x in launches] == [1, 1, 1]


def test_results_of_the_step_are_not(launches):
    a, w = torch.randn(4, 128).bfloat16(), _weight()
    gathered = _weight()
    gathered._ats_z3 = object()
    pitched = torch.nn.Parameter(torch.randn(256, 129).bfloat16()[:, :128], requires_grad=False)   # rows not 16-byte aligned: the product reads a copy
    for fresh in (w * 2, w[:128], gathered, pitched):
        G.gemm_nt(a, fresh)
        G.gemm_nt_swiglu(a, fresh)
    assert [x.w_ready for x in launches] == [0] * 8


@pytest.mark.parametrize("rows", [17, 33, 64])
def test_dequantised_weights_are_not(launches, monkeypatch, rows):
    """More rows than the 4-bit streaming kernel takes: the weight is written out inside the step."""
    wd = torch.randn(256, 512).bfloat16()
    monkeypatch.setattr(int4, "dequantize", lambda *entry: wd)
    a = torch.randn(rows, 512).bfloat16()
    int4._matmul(a, (None, None, 64), None)
    int4._matmul(a, (None, None, 64), None, swiglu=True)
    assert [x.w_ready for x in launches] == [0, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [17, 33, 64])
def test_captured_step_on_4_bit_weights(rows, monkeypatch):
    """Chained launches change the order of nothing: the kernels sum in fixed orders, so the logits of a captured step are equal bit by bit."""
    import contextlib
    from adaptivetrainingsystem_b200.config import ModelConfig
    from adaptivetrainingsystem_b200.inference import engine as E
    from adaptivetrainingsystem_b200.models.transformer import DeepSeekTransformer
    torch.manual_seed(rows)
    cfg = ModelConfig(vocab_size=2048, hidden_size=512, num_layers=3, num_heads=8, num_kv_heads=2, intermediate_size=1024, seq_length=64, tie_word_embeddings=False)
    model = DeepSeekTransformer(cfg).cuda().to(torch.bfloat16).eval()
    ids = torch.randint(0, 2048, (rows, 20), device="cuda")
    try:
        int4.clear()
        for blk in model.layers:
            for w in (blk.self_attn.qkv_proj, blk.self_attn.o_proj, blk.ffn.gate_up_proj, blk.ffn.down_proj):
                int4.register(w.detach())
        int4.set_enabled(True)
        logits = []
        for chained in (True, False):
            if not chained:
                monkeypatch.setattr(E, "chained_launches", lambda on=True: contextlib.nullcontext())
            eng = E.GenerationEngine(model, max_batch=rows)
            cache = model.make_cache(rows, 32)
            with torch.no_grad():
                eng.prefill(ids[:, :8], cache)
                dec = E.GraphDecoder(model, cache)
                logits.append([dec.step(ids[:, 8 + i]).clone() for i in range(12)])
        for a, b in zip(*logits):
            assert bool(torch.isfinite(a.float()).all()) and torch.equal(a, b)
    finally:
        int4.set_enabled(False)
        int4.clear()
