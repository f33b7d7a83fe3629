"""Programmatic dependent launch without further promises: what the launch directly ahead has written is what a kernel reads."""
import math

import pytest
import torch

from gpu_util import native, status_word

pytestmark = pytest.mark.gpu


def bf(*shape):
    return torch.randn(*shape, device="cuda").to(torch.bfloat16)


def swiglu(C, st):
    x, out = bf(16, 1024), torch.empty(16, 4096, device="cuda", dtype=torch.bfloat16)
    return (8192, 1024), lambda w: (C.gemm_swiglu(x, w, out, None, 1e-6, st), out)[1]


def splitk(C, st):
    x, out = bf(16, 1024), torch.empty(16, 8192, device="cuda", dtype=torch.bfloat16)

    def run(w):
        assert C.gemm_decode(x, w, out, None, None, None, None, 1e-6, st)
        return out

    return (8192, 1024), run


def sample(C, st):
    R, V, H = 16, 8192, 1024
    x, seeds = bf(R, H), torch.zeros(R, dtype=torch.int64, device="cuda")
    n = int(C.lm_sample_num_groups(V, R)) * R
    f, i = torch.empty(4 * n, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
    tok, lp = torch.empty(R, dtype=torch.int32, device="cuda"), torch.empty(R, device="cuda")
    return (V, H), lambda w: (C.lm_sample(x, w, 0.0, seeds, f, i, tok, lp, st), torch.stack([tok.float(), lp]))[1]


def attention(C, st):
    B, Hq, Hkv, D, nb = 8, 12, 2, 128, 64
    q, out = bf(B, (Hq + 2 * Hkv) * D), torch.empty(B, Hq * D, device="cuda", dtype=torch.bfloat16)
    v = bf(B * nb, Hkv, 16, D)
    bt = torch.arange(B * nb, dtype=torch.int32, device="cuda").view(B, nb)
    lens = torch.full((B,), nb * 16 - 3, dtype=torch.int32, device="cuda")

    def run(w):
        C.paged_decode_attn(q, w.view(B * nb, Hkv, 16, D), v, bt, lens, out, Hq, Hkv, D, 1 / math.sqrt(D), 1, torch.empty(1, device="cuda"),
                            torch.empty(1, device="cuda"), st, None)
        return out

    return (B * nb * Hkv * 16, D), run


@pytest.mark.parametrize("make", [swiglu, splitk, sample, attention])
def test_operands_written_by_the_launch_ahead(make):
    C, st = native(), status_word()
    torch.manual_seed(0)
    (rows, cols), run = make(C, st)
    ones = torch.ones(cols, device="cuda", dtype=torch.bfloat16)
    srcs = [bf(rows, cols) for _ in range(2)]
    w = torch.empty(rows, cols, device="cuda", dtype=torch.bfloat16)
    want = []
    for s in srcs:
        C.rmsnorm_fwd(s, ones, w, None, 1e-6)
        want.append(run(w).clone())
    assert not torch.equal(*want)
    C.set_pdl(True)
    try:
        got = []
        for k in range(24):
            C.rmsnorm_fwd(srcs[k & 1], ones, w, None, 1e-6)  # lets its successor begin while it still writes
            got.append(run(w).clone())
    finally:
        C.set_pdl(False)
    assert int(st.item()) == 0
    assert all(torch.equal(g, want[k & 1]) for k, g in enumerate(got))
