"""Paged decode attention at the edges of its block pipeline: newest token alone in a block, sequences shorter than the blocks
requested ahead, more than 32 blocks a warp, idle rows."""
import math

import pytest
import torch

from gpu_util import native, status_word

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,splits", [(12, 2, 1), (12, 2, 3), (28, 4, 8), (4, 4, 2)])
def test_paged_decode_attention_block_edges(Hq, Hkv, splits):
    C = native()
    torch.manual_seed(Hq + splits)
    D, bs, dev = 128, 16, "cuda"
    lens_l = [1, 15, 16, 17, 0, 33, 64, 65, 129, 2047, 2049, 4600]
    B, mb = len(lens_l), (max(lens_l) + bs - 1) // bs
    lens = torch.tensor(lens_l, dtype=torch.int32, device=dev)
    nblk = B * mb
    kc, vc = (torch.randn(nblk, Hkv, bs, D, device=dev).to(torch.bfloat16) for _ in range(2))
    bt = torch.randperm(nblk, device=dev).to(torch.int32).view(B, mb).contiguous()
    q = torch.randn(B, (Hq + 2 * Hkv) * D, device=dev).to(torch.bfloat16)
    out = torch.zeros(B, Hq * D, dtype=torch.bfloat16, device=dev)
    po, pm = torch.empty(B * Hkv * splits * 8 * D, device=dev), torch.empty(B * Hkv * splits * 16, device=dev)
    tickets, st = torch.zeros(B * Hkv, dtype=torch.int32, device=dev), status_word()
    C.paged_decode_attn(q, kc, vc, bt, lens, out, Hq, Hkv, D, 1 / math.sqrt(D), splits, po, pm, st, tickets)
    assert int(st.item()) == 0 and int(tickets.abs().max()) == 0
    for b, n in enumerate(lens_l):
        if n == 0:
            continue
        nb = (n + bs - 1) // bs
        k, v = (c[bt[b, :nb].long()].permute(1, 0, 2, 3).reshape(Hkv, nb * bs, D)[:, :n].double() for c in (kc, vc))
        w = torch.softmax(torch.einsum("hgd,hld->hgl", q[b, :Hq * D].view(Hkv, Hq // Hkv, D).double(), k) / math.sqrt(D), -1)
        ref, mag = (torch.einsum("hgl,hld->hgd", w, t).reshape(-1) for t in (v, v.abs()))
        # probabilities and output are rounded to bf16: 8 significant bits, so 2^-8 of a value at most; the rest is fp32
        assert bool(((out[b].double() - ref).abs() <= 2 ** -8 * (mag + ref.abs()) + 1e-5 * mag).all())
