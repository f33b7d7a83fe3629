"""How many columns of the logits a training step may keep for its backward pass."""
from types import SimpleNamespace

import torch

from async_grpo_nccl_b200.models.decoder import NativeDecoder


def test_memory_is_that_of_the_decoders_device():
    asked = []
    dec = SimpleNamespace(dev=torch.device("cuda", 1), cfg=SimpleNamespace(vocab_size=1000), _activation_bytes=lambda T: 7.0 * T,
                          C=SimpleNamespace(lmhead_keep_columns=lambda device, rows, V, reserve: asked.append((device, rows, V, reserve)) or 8))
    assert NativeDecoder._keep_columns(dec, 5, 9) == 8
    assert asked == [(1, 5, 1000, 63.0)]
