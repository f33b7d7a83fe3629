"""Forward and backward over the rows that carry a loss alone, against all rows."""
import numpy as np
import pytest
import torch

from gpu_util import rel_err

pytestmark = pytest.mark.gpu


def samples(lens, vocab, seed=0):
    rng = np.random.default_rng(seed)
    return [{"sample_ids": rng.integers(2, vocab, p + n).astype(np.int32), "input_len": p, "output_len": n, "advantage": float(rng.normal()),
             "sample_logprobs": rng.normal(size=p + n) - 8, "sample_entropies": rng.random(p + n), "ref_logprobs": rng.normal(size=p + n) - 8}
            for p, n in lens]


def run(monkeypatch, pb, min_flops):
    from async_grpo_nccl_b200.models import decoder as D
    from async_grpo_nccl_b200.models.config import PRESETS
    from async_grpo_nccl_b200.models.layout import ParamLayout

    monkeypatch.setattr(D, "LOSS_ROWS_MIN_FLOPS", min_flops)
    cfg = PRESETS["tiny128"]
    layout = ParamLayout(cfg)
    flat = torch.empty(layout.total, dtype=torch.bfloat16, device="cuda")
    layout.init_random_device_(flat, 1)
    dec = D.NativeDecoder(cfg, layout, flat)
    sink = D.GradSink(layout, "cuda")
    stats = dec.forward_backward(pb, D.LossConfig(kl_beta=0.1, temperature=0.9), 0.5, sink)
    dec.check_status()
    return stats, sink.flat


# one output; outputs from the first row on (a prompt of one token); fewer and more than 128 rows with a loss, odd counts; no output
@pytest.mark.parametrize("lens", [[(40, 1)], [(1, 90), (7, 3)], [(130, 60), (1, 129), (33, 0), (5, 77)], [(50, 0)]])
def test_rows_without_a_loss_can_be_left_out(monkeypatch, lens):
    from async_grpo_nccl_b200.packing import pack_samples

    pb = pack_samples(samples(lens, 2000)).to_device("cuda")
    assert pb.loss_rows
    stats0, g0 = run(monkeypatch, pb, 1e30)
    stats1, g1 = run(monkeypatch, pb, -1.0)
    # statistics are fp32 sums over the same rows; the output matrix's gradient sums the same products in another order (fp32), the
    # other gradients see bf16 roundings of the same values and dQ tiles in any order
    torch.testing.assert_close(stats0, stats1, rtol=1e-4, atol=1e-3)
    assert rel_err(g1, g0) < 1e-3


def test_sample_without_prompt_keeps_all_rows():
    from async_grpo_nccl_b200.packing import pack_samples

    assert not pack_samples(samples([(0, 9), (4, 3)], 2000)).loss_rows


# rows below and above one pair tile, a vocabulary that is no multiple of 8, buffers that hold no, some and all of the columns
@pytest.mark.parametrize("T,H,V,chunk,keep", [(70, 128, 1003, 512, 1008), (300, 256, 2048, 512, 2048), (300, 256, 2048, 512, 1280), (513, 128, 5001, 1024, 2048),
                                              (129, 64, 264, 256, 256)])
def test_kept_logits_give_the_same_gradients(T, H, V, chunk, keep):
    from gpu_util import native, status_word

    C = native()
    torch.manual_seed(T)
    h, W = (torch.randn(n, H, device="cuda").mul_(0.3).to(torch.bfloat16) for n in (T, V))
    labels = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
    labels[::7] = -1
    dlogp, st = torch.randn(T, device="cuda"), status_word()
    groups = C.lmhead_num_groups(V, T)
    got = []
    for logits in (None, torch.full((T, keep), float("nan"), device="cuda")):
        f = lambda n: torch.zeros(n, device="cuda")
        logp, ent, lse = f(T), f(T), f(T)
        C.lmhead_logprob(h, W, labels, 0.7, f(3 * groups * T), f(T), logp, ent, lse, st, logits)
        dz, dh, dW = torch.empty(T, chunk, device="cuda", dtype=torch.bfloat16), f(T * H).view(T, H), f(V * H).view(V, H)
        C.lmhead_backward(h, W, labels, lse, dlogp, 0.7, dz, dh, dW, st, logits)
        got.append((logp, ent, lse, dh, dW))
    assert int(st.item()) == 0
    assert all(torch.equal(a, b) for a, b in zip(*got))
