"""Training steps with none, some and all of their logits kept, and at the limit of the memory."""
import dataclasses

import numpy as np
import pytest
import torch

from gpu_util import native, rel_err

pytestmark = pytest.mark.gpu


def decoder(model, layers, recompute=False):
    from async_grpo_nccl_b200.models import decoder as D
    from async_grpo_nccl_b200.models.config import PRESETS
    from async_grpo_nccl_b200.models.layout import ParamLayout

    cfg = dataclasses.replace(PRESETS[model], num_hidden_layers=layers)
    layout = ParamLayout(cfg)
    flat = torch.empty(layout.total, dtype=torch.bfloat16, device="cuda")
    layout.init_random_device_(flat, 1)
    return D.NativeDecoder(cfg, layout, flat, recompute=recompute), D.GradSink(layout, "cuda")


def batch(lens, vocab):
    from async_grpo_nccl_b200.packing import pack_samples

    rng = np.random.default_rng(len(lens))
    return pack_samples([{"sample_ids": rng.integers(2, vocab, p + n).astype(np.int32), "input_len": p, "output_len": n, "advantage": float(rng.normal()),
                          "sample_logprobs": rng.normal(size=p + n) - 8, "sample_entropies": rng.random(p + n)} for p, n in lens]).to_device("cuda")


def step(dec, sink, pb):
    from async_grpo_nccl_b200.models.decoder import LossConfig

    sink.zero_()
    stats = dec.forward_backward(pb, LossConfig(), 1.0, sink)
    dec.check_status()
    return stats, sink.flat.cpu()


@pytest.mark.parametrize("recompute", [False, True])
def test_a_step_that_fits_without_kept_logits_still_fits(monkeypatch, recompute):
    dec, sink = decoder("qwen2.5-1.5b", 2, recompute)
    pb = batch([(9, 1700), (200, 1400), (3, 700)], 150000)  # logits of 2.3 GB, a quarter of what else the step holds
    # what the head's products keep beside torch's allocator is there before the limit is
    with monkeypatch.context() as m:
        m.setattr(type(dec), "_keep_columns", lambda *a: 0)
        want = step(dec, sink, pb)
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        step(dec, sink, pb)
        peak = torch.cuda.max_memory_reserved()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((peak + (256 << 20)) / total)
        for _ in range(3):
            got = step(dec, sink, pb)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    torch.testing.assert_close(got[0], want[0], rtol=1e-4, atol=1e-3)
    # the output matrix's gradient has the same bits with and without kept logits; dQ tiles are added in any order (bf16 after them)
    assert rel_err(got[1], want[1]) < 1e-3


@pytest.mark.parametrize("V_kept", [0, 256, 60160, 151936])
def test_columns_kept_do_not_change_the_gradients(monkeypatch, V_kept):
    dec, sink = decoder("qwen2.5-1.5b", 1)
    pb = batch([(9, 130), (40, 77)], 150000)
    results = []
    for keep in (0, V_kept):
        monkeypatch.setattr(type(dec), "_keep_columns", lambda *a: keep)
        stats, grads = step(dec, sink, pb)
        results.append((stats, dec.layout.view(grads, "final_norm").clone(), grads))
    # statistics and the final norm's gradient are summed atomically (fp32, any order)
    torch.testing.assert_close(results[0][0], results[1][0], rtol=1e-5, atol=1e-4)
    torch.testing.assert_close(results[0][1], results[1][1], rtol=1e-4, atol=1e-6)
    assert rel_err(results[1][2], results[0][2]) < 1e-3


def test_the_same_step_finds_what_it_has_left(monkeypatch):
    dec, sink = decoder("qwen2.5-1.5b", 4)
    torch.cuda.empty_cache()
    asked, kept = [], []
    info, keep = torch.cuda.mem_get_info, type(dec)._keep_columns
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d=None: asked.append(d) or info(d))
    monkeypatch.setattr(type(dec), "_keep_columns", lambda *a: kept.append(keep(*a)) or kept[-1])
    for lens in ([(9, 3000), (200, 1400)], [(9, 3000), (200, 1400)], [(3, 2900), (100, 1000)], [(1, 5000)], [(1, 5000)], [(9, 3000), (200, 1400)]):
        step(dec, sink, batch(lens, 150000))
    assert kept == [151936] * 6 and len(asked) <= 2  # the first and the larger one


def test_cached_memory_is_that_of_the_stream():
    C = native()
    torch.cuda.empty_cache()
    piece, big = 1 << 20, 256 << 20
    before, block, held = C.cached_memory(0, piece)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        t = torch.empty(big, dtype=torch.uint8, device="cuda")
        assert C.cached_memory(0, piece) == (0, 0, held + big)
        del t
        assert C.cached_memory(0, piece) == (big, big, held + big)
    assert C.cached_memory(0, piece) == (before, block, held + big)  # not of this one
    a = torch.empty(big + (64 << 20), dtype=torch.uint8, device="cuda")
    del a
    b = torch.empty(big, dtype=torch.uint8, device="cuda")  # out of the block of a: what is left of it counts in whole pieces
    assert C.cached_memory(0, 48 << 20)[0] - C.cached_memory(0, 1 << 40)[0] >= 48 << 20
    del b
    torch.cuda.empty_cache()
