"""Attention backward with the rotary embedding undone on the way out."""
import pytest
import torch

from gpu_util import make_tiles, native, rel_err, status_word

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [64, 128])
def test_attention_backward_rotates(D):
    """Against the separate rotation kernel, which rounds to bf16 once more (2^-9 of each value)."""
    C, st = native(), status_word()
    torch.manual_seed(D)
    lens, Hq, Hkv = [1, 130, 300], 6, 2
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
    assert torch.equal(got[:, (Hq + Hkv) * D:], want[:, (Hq + Hkv) * D:])
    C.rope_inplace(want, pos, cos_t, sin_t, Hq + Hkv, D, True)
    assert int(st.item()) == 0
    assert rel_err(got.double(), want.double()) < 2.0 ** -8
