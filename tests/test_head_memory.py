"""What the output head of a training step holds, and that the memory estimate counts it."""
import pytest

from adaptivetrainingsystem_b200 import ops
from adaptivetrainingsystem_b200.config import ConfigPresets


@pytest.mark.parametrize("rows,vocab,width", [(16384, 32000, 2048), (4096, 200000, 4096), (16777, 32000, 1024), (16778, 32000, 1024), (65536, 32000, 4096)])
def test_head_bytes(rows, vocab, width):
    kept = rows <= ops.head_chunk_rows(vocab)
    assert kept == (rows <= 4096 or 2 * rows * vocab <= 1 << 30)
    # gradients of all logits until the backward pass, or those of 4,096 rows beside fp32 sums of the weight gradient
    assert ops.head_bytes(rows, vocab, width) == (2 * rows * vocab if kept else 2 * 4096 * vocab + 4 * vocab * width)


@pytest.mark.parametrize("micro_batch", [1, 8, 64])
def test_memory_estimate_counts_the_head(micro_batch):
    cfg = ConfigPresets.get("dense_1b", micro_batch_size=micro_batch, batch_size=micro_batch)
    tokens = micro_batch * cfg.seq_length
    layers = tokens * cfg.hidden_size * 2 * (2 if cfg.gradient_checkpointing else 18) * cfg.num_layers
    held = cfg.get_memory_estimate_gb()["activations"] * 1024 ** 3 - layers
    assert held == pytest.approx(ops.head_bytes(tokens, cfg.vocab_size, cfg.hidden_size), rel=1e-6)
