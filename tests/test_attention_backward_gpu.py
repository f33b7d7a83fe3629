"""Attention backward with the rotary embedding undone on the way out."""
import pytest
import torch

from gpu_util import make_tiles, native, rel_err, status_word

pytestmark = pytest.mark.gpu
DEV = "cuda"


# several CTAs per kv head: dK is rotated where their parts are summed; one (Hq == Hkv): in the kernel itself
@pytest.mark.parametrize("Hq,Hkv", [(6, 2), (2, 2)])
@pytest.mark.parametrize("D", [64, 128])
def test_attention_backward_rotates(D, Hq, Hkv):
    """Against the separate rotation kernel, which rounds to bf16 once more (2^-9 of each value)."""
    C, st = native(), status_word()
    torch.manual_seed(D)
    lens = [1, 130, 300]
    T, cols = sum(lens), (Hq + 2 * Hkv) * D
    qkv = torch.randn(T, cols, device=DEV).to(torch.bfloat16)
    dout = torch.randn(T, Hq * D, device=DEV).to(torch.bfloat16)
    out, lse = torch.empty_like(dout), torch.empty(Hq, T, device=DEV)
    tiles, sc = make_tiles(lens), D ** -0.5
    C.attn_varlen_fwd(qkv, out, lse, tiles, Hq, Hkv, D, sc, st)
    pos = torch.cat([torch.arange(n, dtype=torch.int32) for n in lens]).to(DEV)
    ang = torch.randn(256, D // 2, device=DEV)  # positions 256 .. use the last row
    cos_t, sin_t = ang.cos().contiguous(), ang.sin().contiguous()
    delta, acc = torch.empty(Hq, T, device=DEV), torch.empty(T, Hq * D, device=DEV)
    got, want = (torch.zeros(T, cols, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    C.attn_varlen_bwd(qkv, out, dout, lse, delta, acc, got, tiles, Hq, Hkv, D, sc, st, pos, cos_t, sin_t)
    C.attn_varlen_bwd(qkv, out, dout, lse, delta, acc, want, tiles, Hq, Hkv, D, sc, st)
    assert (C.attn_bwd_pieces(tiles.shape[0], Hq, Hkv) == 1) == (Hq == Hkv)
    assert torch.equal(got[:, (Hq + Hkv) * D:], want[:, (Hq + Hkv) * D:])  # dV is not rotated
    C.rope_inplace(want, pos, cos_t, sin_t, Hq + Hkv, D, True)
    assert int(st.item()) == 0
    assert rel_err(got.double(), want.double()) < 2.0 ** -8


# 1 key tile per head: as many CTAs as query heads; 7 heads in 7, in 2 (100 tiles x 4 kv heads) and in 1 piece (600 x 4)
@pytest.mark.parametrize("lens,Hq,Hkv,D", [([5, 128], 6, 2, 128), ([300, 129, 1], 7, 1, 64), ([128] * 100, 28, 4, 128), ([40] * 600, 28, 4, 64)])
def test_attention_backward_pieces(lens, Hq, Hkv, D):
    """Query heads of a group dealt to several CTAs, against fp64; dK and dV repeat bit for bit."""
    C, st = native(), status_word()
    torch.manual_seed(len(lens))
    T, cols, g = sum(lens), (Hq + 2 * Hkv) * D, Hq // Hkv
    qkv = torch.randn(T, cols, device=DEV).to(torch.bfloat16)
    dout = torch.randn(T, Hq * D, device=DEV).to(torch.bfloat16)
    out, lse = torch.empty_like(dout), torch.empty(Hq, T, device=DEV)
    tiles, sc = make_tiles(lens), D ** -0.5
    C.attn_varlen_fwd(qkv, out, lse, tiles, Hq, Hkv, D, sc, st)
    delta, acc = torch.empty(Hq, T, device=DEV), torch.empty(T, Hq * D, device=DEV)
    got = torch.zeros(T, cols, device=DEV, dtype=torch.bfloat16)
    C.attn_varlen_bwd(qkv, out, dout, lse, delta, acc, got, tiles, Hq, Hkv, D, sc, st)
    assert int(st.item()) == 0
    for _ in range(4):
        again = torch.zeros_like(got)
        C.attn_varlen_bwd(qkv, out, dout, lse, delta, acc, again, tiles, Hq, Hkv, D, sc, st)
        assert torch.equal(again[:, Hq * D:], got[:, Hq * D:])
    x = qkv.double().requires_grad_(True)
    h, o, outs = x.view(T, Hq + 2 * Hkv, D), 0, []
    for n in lens:
        q, k, v = (h[o:o + n, a:b].transpose(0, 1) for a, b in ((0, Hq), (Hq, Hq + Hkv), (Hq + Hkv, Hq + 2 * Hkv)))
        k, v = k.repeat_interleave(g, 0), v.repeat_interleave(g, 0)
        z = (q @ k.transpose(1, 2) * sc).masked_fill(torch.ones(n, n, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
        outs.append((torch.softmax(z, -1) @ v).transpose(0, 1).reshape(n, Hq * D))
        o += n
    torch.cat(outs).backward(dout.double())
    # P and dS are bf16 operands (2^-9 each), the result is bf16: a few 2^-9 of the gradient's size
    for a, b in ((0, Hq * D), (Hq * D, (Hq + Hkv) * D), ((Hq + Hkv) * D, cols)):
        assert rel_err(got[:, a:b].double(), x.grad[:, a:b]) < 2e-2


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("Hq,Hkv,D", [(2, 2, 128), (2, 2, 64), (6, 2, 128), (6, 2, 64)])
def test_attention_backward_keeps_sequences_apart(Hq, Hkv, D, bad):
    """A sequence whose last rows are not finite: the gradients of the sequence after it, whose first rows share its tiles, are
    bit for bit those without, with one CTA per kv head and with several."""
    C, st = native(), status_word()
    torch.manual_seed(D)
    lens, cols = [100, 120], (Hq + 2 * Hkv) * D
    T, n = sum(lens), lens[0]
    clean = torch.randn(T, cols, device=DEV).to(torch.bfloat16)
    clean_dout = torch.randn(T, Hq * D, device=DEV).to(torch.bfloat16)
    tiles, sc, grads = make_tiles(lens), D ** -0.5, []
    for poison in (False, True):
        qkv, dout = clean.clone(), clean_dout.clone()
        if poison:
            qkv[n - 2], dout[n - 2] = bad, bad
        out, lse = torch.empty_like(dout), torch.empty(Hq, T, device=DEV)
        C.attn_varlen_fwd(qkv, out, lse, tiles, Hq, Hkv, D, sc, st)
        assert (C.attn_bwd_pieces(tiles.shape[0], Hq, Hkv) > 1) == (Hq > Hkv)
        delta, acc, got = torch.empty(Hq, T, device=DEV), torch.empty(T, Hq * D, device=DEV), torch.zeros(T, cols, device=DEV, dtype=torch.bfloat16)
        C.attn_varlen_bwd(qkv, out, dout, lse, delta, acc, got, tiles, Hq, Hkv, D, sc, st)
        grads.append(got)
    assert int(st.item()) == 0
    assert bool(grads[0].isfinite().all()) and not bool(grads[1][:n].isfinite().all())
    assert torch.equal(grads[1][n:], grads[0][n:])


@pytest.mark.parametrize("Hq,Hkv", [(2, 2), (6, 2)])
def test_attention_backward_writes_rows_of_its_tiles(Hq, Hkv):
    """Rows that belong to no tile: dK and dV stay as they were, with one CTA per kv head and with several."""
    C, st, D = native(), status_word(), 64
    torch.manual_seed(Hq)
    lens, rest = [130, 40], 50
    T, cols = sum(lens) + rest, (Hq + 2 * Hkv) * D
    qkv = torch.randn(T, cols, device=DEV).to(torch.bfloat16)
    dout = torch.randn(T, Hq * D, device=DEV).to(torch.bfloat16)
    out, lse, tiles = torch.zeros_like(dout), torch.zeros(Hq, T, device=DEV), make_tiles(lens)
    C.attn_varlen_fwd(qkv, out, lse, tiles, Hq, Hkv, D, D ** -0.5, st)
    delta, acc = torch.empty(Hq, T, device=DEV), torch.empty(T, Hq * D, device=DEV)
    got = torch.full((T, cols), 7.0, device=DEV, dtype=torch.bfloat16)
    C.attn_varlen_bwd(qkv, out, dout, lse, delta, acc, got, tiles, Hq, Hkv, D, D ** -0.5, st)
    assert int(st.item()) == 0
    assert bool((got[-rest:, Hq * D:] == 7.0).all()) and bool((got[-rest:, :Hq * D] == 0.0).all())
    assert not bool((got[:-rest] == 7.0).all(1).any())
