"""How many columns of the logits a training step may keep for its backward pass."""
from types import SimpleNamespace

import pytest
import torch

from async_grpo_nccl_b200.models import decoder as D
from async_grpo_nccl_b200.ops import native

GB = 1 << 30


class Memory:
    """A decoder's view of a device: ``cached`` bytes unused in the allocator, ``free`` on the device, ``fraction`` and ``share`` allowed."""

    def __init__(self, monkeypatch, cached, reserved, free, held=30 * GB, V=151936, total=180 * GB, fraction=1.0, share=1.0):
        self.asked, self.block = [], None
        self.dec = SimpleNamespace(dev=torch.device("cuda", 1), cfg=SimpleNamespace(vocab_size=V, hidden_size=1536), _asked_at=-1, memory_share=share,
                                   _held_bytes=lambda T, rows: held, C=SimpleNamespace(cached_memory=self.cached_memory, lmhead_chunk_step=native().lmhead_chunk_step),
                                   _chunk=lambda rows: 15360)
        self.cached, self.reserved, self.free, self.total = cached, reserved, free, total
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
        monkeypatch.setattr(torch.cuda, "mem_get_info", self.mem_get_info)
        monkeypatch.setattr(torch.cuda, "get_per_process_memory_fraction", lambda dev: fraction)

    def cached_memory(self, device, piece):
        assert device == 1 and piece > 0
        return self.cached, self.block if self.block is not None else self.cached, self.reserved

    def mem_get_info(self, dev):
        assert dev == torch.device("cuda", 1)
        self.asked.append(dev)
        return self.free, self.total

    def keep(self, rows, T):
        return D.NativeDecoder._keep_columns(self.dec, rows, T)


def test_columns_that_fit():
    assert D.kept_columns(100, 1003, 100 * 4 * 1008, 256) == 1008
    assert D.kept_columns(100, 1003, 100 * 4 * 1008 - 1, 256) == 768
    assert D.kept_columns(100, 1003, 100 * 4 * 255, 256) == 0
    assert D.kept_columns(100, 1003, -5.0, 256) == 0


# the fewest chunks of equal width (a multiple of 256) that the buffer allows
@pytest.mark.parametrize("V,chunk,step", [(151936, 15360, 15360), (152064, 15360, 15360), (2048, 2048, 2048), (1003, 512, 512), (5001, 2048, 1792),
                                          (100, 256, 256), (256, 256, 256), (257, 256, 256)])
def test_steps_of_the_backward_pass(V, chunk, step):
    assert native().lmhead_chunk_step(V, chunk) == step
    for memory in (0, 3 << 20, 40 << 20, 1 << 40):
        kept = D.kept_columns(1000, V, memory, step)
        assert kept % step == 0 or kept == (V + 7) // 8 * 8


@pytest.mark.parametrize("cached,free", [(40, 0), (33, 9), (31, 0), (30, 50)])
def test_only_columns_that_are_read_are_kept(monkeypatch, cached, free):
    m = Memory(monkeypatch, cached * GB, 60 * GB, free * GB)
    cols = m.keep(30000, 32768)
    assert cols % 15360 == 0 and cols < 151936


# need: 30000 x 151936 x 4 = 17.0 GB beside 72 GB that the step holds anyway. A cache filled by a larger microbatch without kept logits
# has room for the step, not for all of its logits: what is short would be an activation's.
@pytest.mark.parametrize("cached,all_kept", [(72 + 17, True), (85, False), (73, False), (60, False)])
def test_cached_memory_must_hold_the_step_and_the_logits(monkeypatch, cached, all_kept):
    m = Memory(monkeypatch, cached * GB, 120 * GB, 0, held=72 * GB)
    cols = m.keep(30000, 32768)
    assert (cols == 151936) == all_kept
    assert cols * 30000 * 4 <= max(0, cached - 72) * GB


def test_device_is_asked_again_only_after_the_allocator_has_changed(monkeypatch):
    m = Memory(monkeypatch, 33 * GB, 40 * GB, 20 * GB)
    first = m.keep(30000, 32768)
    assert len(m.asked) == 1 and 0 < first * 120000 <= 23 * GB // 4
    m.cached, m.reserved = 36 * GB, 43 * GB
    m.keep(30000, 32768)
    assert len(m.asked) == 2
    again = m.keep(30000, 32768)
    assert len(m.asked) == 2 and again * 120000 <= 6 * GB
    m.cached = 60 * GB  # all of it from here on
    assert m.keep(30000, 32768) == 151936 and len(m.asked) == 2


def test_one_block_holds_the_logits(monkeypatch):
    m = Memory(monkeypatch, 60 * GB, 70 * GB, 0)
    m.block = 5 * GB  # the rest in smaller ones: a larger block would come from the device, which has nothing left
    assert 0 < m.keep(30000, 32768) * 120000 <= 5 * GB
    m.dec._asked_at, m.free = -1, 100 * GB
    assert m.keep(30000, 32768) == 151936
    m.dec._asked_at, m.free, m.cached = -1, 25 * GB, 28 * GB  # the activations take 2 GB of it
    assert 0 < m.keep(30000, 32768) * 120000 <= 23 * GB // 4


@pytest.mark.parametrize("kw", [dict(fraction=0.25), dict(share=0.5)])
def test_limits_of_the_process(monkeypatch, kw):
    # 90 GB free on the device, 45 GB held: a process limit of 45 GB, or a share of the device that others have left half used
    m = Memory(monkeypatch, 31 * GB, 45 * GB, 90 * GB, **kw)
    assert m.keep(30000, 32768) * 120000 <= 1 * GB


def test_nothing_is_kept_without_rows_or_in_a_graph(monkeypatch):
    m = Memory(monkeypatch, 100 * GB, 120 * GB, 0)
    assert m.keep(0, 100) == 0
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert m.keep(100, 100) == 0
