"""How many columns of the logits a training step may keep for its backward pass."""
from types import SimpleNamespace

import pytest
import torch

from async_grpo_nccl_b200.models import decoder as D
from async_grpo_nccl_b200.ops import native

GB = 1 << 30
ROWS, V = 30000, 151936
NEED = ROWS * V * 4               # 17 GB
HEAD = ROWS * (2 * 15360 + 6 * 1536)  # 1.1 GB


class Memory:
    """A decoder's view of a device: ``cached`` bytes unused in the allocator (the largest block ``block``), ``free`` on the device,
    ``fraction`` and ``share`` allowed."""

    def __init__(self, monkeypatch, cached, reserved, free, total=180 * GB, fraction=1.0, share=1.0):
        self.asked, self.block = [], None
        self.dec = SimpleNamespace(dev=torch.device("cuda", 1), cfg=SimpleNamespace(vocab_size=V, hidden_size=1536), _asked=(-1, 0), memory_share=share,
                                   C=SimpleNamespace(cached_memory=self.cached_memory, lmhead_chunk_step=native().lmhead_chunk_step),
                                   _chunk=lambda rows: 15360)
        self.cached, self.reserved, self.free, self.total = cached, reserved, free, total
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
        monkeypatch.setattr(torch.cuda, "get_allocator_backend", lambda: "native")
        monkeypatch.setattr(torch.cuda, "mem_get_info", self.mem_get_info)
        monkeypatch.setattr(torch.cuda, "get_per_process_memory_fraction", lambda dev: fraction)

    def cached_memory(self, device, piece):
        assert device == 1 and piece > 0
        return self.cached, self.block if self.block is not None else self.cached, self.reserved

    def mem_get_info(self, dev):
        assert dev == self.dec.dev
        self.asked.append(dev)
        return self.free, self.total

    def keep(self, rows=ROWS):
        cols = D.NativeDecoder._keep_columns(self.dec, rows)
        assert cols == V or cols % 15360 == 0  # only columns that are read
        return cols

    def bytes(self):
        return self.keep() * 4 * ROWS


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


@pytest.mark.parametrize("cached", [0, HEAD, HEAD + NEED // 2, HEAD + NEED - 1, HEAD + NEED])
def test_the_allocator_must_hold_the_logits_and_the_head(monkeypatch, cached):
    m = Memory(monkeypatch, cached, 120 * GB, 0)
    assert (m.keep() == V) == (cached >= HEAD + NEED) and m.bytes() <= max(0, cached - HEAD)


def test_device_is_asked_again_only_after_the_allocator_has_changed(monkeypatch):
    m = Memory(monkeypatch, 4 * GB, 40 * GB, 20 * GB)
    first = m.bytes()
    assert len(m.asked) == 1 and 0 < first <= (24 * GB - HEAD) // 4
    m.cached, m.reserved = 9 * GB, 45 * GB
    m.keep()
    assert len(m.asked) == 2
    assert 0 < m.bytes() <= 9 * GB and len(m.asked) == 2  # one cached block, the head from the device
    m.cached = 40 * GB  # all of it from here on
    assert m.keep() == V and len(m.asked) == 2


def test_one_block_holds_the_logits(monkeypatch):
    m = Memory(monkeypatch, 60 * GB, 70 * GB, 0)
    m.block = 5 * GB  # the rest in smaller ones: a larger block would come from the device, which has nothing left
    assert 0 < m.bytes() <= 5 * GB
    m.dec._asked, m.free = (-1, 0), 100 * GB
    assert m.keep() == V
    m.dec._asked, m.free, m.cached, m.block = (-1, 0), 9 * GB, 0, 0  # the head takes 1.1 GB of it
    assert 0 < m.bytes() <= (9 * GB - HEAD) // 4


@pytest.mark.parametrize("kw", [dict(fraction=0.25), dict(share=0.5)])
def test_limits_of_the_process(monkeypatch, kw):
    # 90 GB free on the device, 45 GB held: a process limit of 45 GB, or a share of the device that others have left half used
    m = Memory(monkeypatch, 5 * GB, 45 * GB, 90 * GB, **kw)
    assert 0 < m.bytes() <= 5 * GB - HEAD


def test_device_without_an_index_is_the_current_one(monkeypatch):
    m = Memory(monkeypatch, 5 * GB, 45 * GB, 9 * GB)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    m.dec.dev = torch.device("cuda")
    assert m.keep() > 0 and len(m.asked) == 1


def test_nothing_is_kept_without_rows_in_a_graph_or_with_another_allocator(monkeypatch):
    m = Memory(monkeypatch, 100 * GB, 120 * GB, 0)
    assert m.keep(0) == 0
    with monkeypatch.context() as other:
        other.setattr(torch.cuda, "get_allocator_backend", lambda: "cudaMallocAsync")
        assert m.keep() == 0
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert m.keep(100) == 0
