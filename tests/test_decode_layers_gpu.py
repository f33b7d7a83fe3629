"""The persistent decode-layers kernel (all decoder layers of one decode step in one launch) against a plain PyTorch
fp32 restatement of the same layers: folded RMSNorm, qkv + bias + RoPE + paged-KV write, GQA attention over the cache,
o-projection + residual, gate/up + SwiGLU, down-projection + residual."""
import math

import pytest
import torch

from gpu_util import native, rel_err, status_word

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _reference(x, Wq, Wo, Wgu, Wd, bq, cache, bt, lens, cos_t, sin_t, Hq, Hkv, eps):
    """fp32 math with bf16 rounding where the kernels store bf16 (activations between GEMMs, cache entries)."""
    L, D, bs = Wq.shape[0], 128, 16
    B, H = x.shape
    F = Wd.shape[2]
    G = Hq // Hkv
    r = lambda t: t.to(torch.bfloat16).float()
    x = x.float()
    kc, vc = cache[:, 0].clone(), cache[:, 1].clone()
    for l in range(L):
        rs = torch.rsqrt((x * x).sum(-1, keepdim=True) / H + eps)
        qkv = rs * (x @ Wq[l].float().t()) + bq[l].float()
        qkv = qkv.view(B, Hq + 2 * Hkv, D)
        pos = (lens.long() - 1).clamp(min=0)
        c, s = cos_t[pos][:, None, :], sin_t[pos][:, None, :]
        rot = qkv[:, :Hq + Hkv]
        x1_, x2_ = rot[..., :64], rot[..., 64:]
        qkv = torch.cat([torch.cat([x1_ * c - x2_ * s, x2_ * c + x1_ * s], -1), qkv[:, Hq + Hkv:]], 1)
        qkv = r(qkv)
        attn = torch.zeros(B, Hq, D, device=x.device)
        for b in range(B):
            n = int(lens[b])
            if n == 0:
                continue
            blk, off = int(bt[b, (n - 1) // bs]), (n - 1) % bs
            kc[l, blk, :, off] = qkv[b, Hq:Hq + Hkv].to(torch.bfloat16)
            vc[l, blk, :, off] = qkv[b, Hq + Hkv:].to(torch.bfloat16)
            nb = (n + bs - 1) // bs
            k = kc[l][bt[b, :nb].long()].permute(1, 0, 2, 3).reshape(Hkv, nb * bs, D)[:, :n].float()
            v = vc[l][bt[b, :nb].long()].permute(1, 0, 2, 3).reshape(Hkv, nb * bs, D)[:, :n].float()
            q = qkv[b, :Hq].view(Hkv, G, D)
            p = torch.softmax(torch.einsum("hgd,hld->hgl", q, k) / math.sqrt(D), -1)
            attn[b] = torch.einsum("hgl,hld->hgd", p, v).reshape(Hq, D)
        attn = r(attn.reshape(B, Hq * D))
        x1 = x + attn @ Wo[l].float().t()
        rs1 = torch.rsqrt((x1 * x1).sum(-1, keepdim=True) / H + eps)
        x1 = r(x1)
        gu = rs1 * (x1 @ Wgu[l].float().t())
        act = r(torch.nn.functional.silu(gu[:, :F]) * gu[:, F:])
        x = r(x1 + act @ Wd[l].float().t())
    return x, kc, vc


@pytest.mark.parametrize("B,H,Hq,Hkv,F,L,splits", [(5, 512, 4, 2, 1408, 2, 1), (32, 512, 4, 2, 1408, 3, 2), (48, 1536, 12, 2, 8960, 2, 2),
                                                   (100, 512, 4, 2, 1408, 2, 1), (200, 1536, 12, 2, 8960, 1, 1)])
def test_decode_layers_match_layer_math(B, H, Hq, Hkv, F, L, splits):
    C = native()
    torch.manual_seed(B + L)
    D, bs, eps = 128, 16, 1e-6
    Q, QD = (Hq + 2 * Hkv) * D, Hq * D
    assert C.decode_layers_supported(B, H, Q, QD, F, Hq, Hkv, D)
    bf = dict(device=DEV, dtype=torch.bfloat16)
    sc = 0.5 / math.sqrt(H)
    Wq = (torch.randn(L, Q, H, device=DEV) * sc).to(torch.bfloat16)
    Wo = (torch.randn(L, H, QD, device=DEV) * sc).to(torch.bfloat16)
    Wgu = (torch.randn(L, 2 * F, H, device=DEV) * sc).to(torch.bfloat16)
    Wd = (torch.randn(L, H, F, device=DEV) * (0.5 / math.sqrt(F))).to(torch.bfloat16)
    bq = (torch.randn(L, Q, device=DEV) * 0.1).to(torch.bfloat16)
    rows = 32 if B <= 32 else 64 if B <= 64 else 128 if B <= 128 else 256
    x = torch.zeros(rows, H, **bf)
    x[:B] = torch.randn(B, H, device=DEV).to(torch.bfloat16)
    x0 = x[:B].clone()
    lens = torch.randint(1, 700, (B,), device=DEV, dtype=torch.int32)
    lens[0] = 0  # an idle row
    max_blocks = 48
    nblk = int(((lens + bs - 1) // bs).sum()) + 4
    cache = (torch.randn(L, 2, nblk, Hkv, bs, D, device=DEV) * 0.5).to(torch.bfloat16)
    perm = torch.randperm(nblk, device=DEV).to(torch.int32)
    bt = torch.full((B, max_blocks), -1, device=DEV, dtype=torch.int32)
    pi = 0
    for b in range(B):
        nb = (int(lens[b]) + bs - 1) // bs
        bt[b, :nb] = perm[pi:pi + nb]
        pi += nb
    max_pos = 1024
    inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, device=DEV).float() / D))
    ang = torch.arange(max_pos, device=DEV).float()[:, None] * inv[None, :]
    cos_t, sin_t = ang.cos().contiguous(), ang.sin().contiguous()
    ref_x, ref_k, ref_v = _reference(x0, Wq, Wo, Wgu, Wd, bq, cache, bt, lens, cos_t, sin_t, Hq, Hkv, eps)

    x1, qkv = torch.zeros(rows, H, **bf), torch.zeros(rows, Q, **bf)
    attn, act = torch.zeros(rows, QD, **bf), torch.zeros(rows, F, **bf)
    ss = torch.zeros(2 * L + 1, rows, device=DEV, dtype=torch.int64)
    ss[0, :B] = ((x0.double() ** 2).sum(-1) * 2 ** 30).round().to(torch.int64)
    part_o = torch.empty(B * Hkv * splits * 8 * D, device=DEV)
    part_ml = torch.empty(B * Hkv * splits * 16, device=DEV)
    tickets = torch.zeros(B * Hkv, device=DEV, dtype=torch.int32)
    partials = torch.empty(C.decode_layers_scratch_bytes(B, H, Q, QD, F) // 4, device=DEV)
    counters = torch.zeros(C.decode_layers_counter_words(), device=DEV, dtype=torch.int32)
    st = status_word()
    for rep in range(2):  # the second call starts from what the first one left behind
        kcache = cache.clone()
        x[:B] = x0
        ss.zero_()
        ss[0, :B] = ((x0.double() ** 2).sum(-1) * 2 ** 30).round().to(torch.int64)
        C.decode_layers(L, B, Wq[0], Q * H, Wo[0], H * QD, Wgu[0], 2 * F * H, Wd[0], H * F, bq[0], Q, x, x1, qkv, attn, act, ss, eps,
                        cos_t, sin_t, bt, lens, kcache, Hq, Hkv, 1 / math.sqrt(D), splits, part_o, part_ml, tickets, partials,
                        counters, st)
        torch.cuda.synchronize()
        assert int(st.item()) == 0
        live = lens > 0
        assert rel_err(x[:B][live], ref_x[live]) < 3e-2
        assert rel_err(kcache[:, 0], ref_k.float()) < 2e-2 and rel_err(kcache[:, 1], ref_v.float()) < 2e-2
        # every partial sum that was handed over has been read, and its word put back to "not yet"
        assert all(bool((t.view(torch.int32) == -1).all()) for t in (partials, part_o, part_ml)[:3 if splits > 1 else 1])
        if rep == 0:
            first = x[:B].clone()
        else:
            assert torch.equal(first, x[:B]), "the reduction order is fixed: two runs give the same bits"
