"""GEMMs on CTA pairs: ragged edges of the 256-row and 256 / 192 / 128-column tiles, each epilogue, against fp64 products of the
same bf16 operands."""
import pytest
import torch

from gpu_util import native, rel_err, status_word

pytestmark = pytest.mark.gpu
DEV = "cuda"
# an fp32 sum of K products: K * 2^-24 relative to the sum of magnitudes, sqrt(K) of it seen; a bf16 result adds 2^-9
F32_TOL, BF16_TOL = 2e-5, 2.0 ** -8


def _operands(M, N, K, a_mn, b_mn):
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV).to(torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV).to(torch.bfloat16)
    return a, b, (a.t() if a_mn else a).double() @ (b.t() if b_mn else b).double().t()


# 129 rows: the second CTA holds one row; 400, 600: one CTA of the last pair is empty or nearly so; 6223 x 1536 takes 192-wide
# tiles, 1536 x 1536 128-wide ones, 3000 x 8960 256-wide ones; widths that end inside a tile and inside a warp's 32 columns
@pytest.mark.parametrize("M,N,K", [(129, 16, 64), (264, 208, 72), (400, 272, 200), (600, 1168, 136), (6223, 1536, 256), (1536, 1536, 520), (3000, 8960, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_pair_gemm(M, N, K, a_mn, b_mn):
    if a_mn and M % 8:
        pytest.skip("an MN-major operand needs a row pitch that is a multiple of 8")
    C, st = native(), status_word()
    torch.manual_seed(M + N)
    a, b, want = _operands(M, N, K, a_mn, b_mn)
    bias = torch.randn(N, device=DEV).to(torch.bfloat16)
    res = torch.randn(M, N, device=DEV).to(torch.bfloat16)
    guard = torch.full((M + 1, N), 7.0, device=DEV, dtype=torch.bfloat16)  # nothing past the last row is written
    C.gemm_bf16(a, b, guard[:M], a_mn, b_mn, None, 1.0, False, st, None)
    assert rel_err(guard[:M].double(), want) < BF16_TOL and bool((guard[M] == 7.0).all())
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    C.gemm_bf16(a, b, out, a_mn, b_mn, bias, 1.0, False, st, res)
    assert rel_err(out.double(), want + bias.double() + res.double()) < BF16_TOL
    acc = torch.randn(M, N, device=DEV)
    total = acc.double() + want
    C.gemm_bf16(a, b, acc, a_mn, b_mn, None, 1.0, True, st, None)
    assert rel_err(acc.double(), total) < F32_TOL
    # a pitch that no 32-byte access fits takes the plain kernel
    odd = torch.empty(M, N + 8, device=DEV, dtype=torch.bfloat16)[:, :N]
    C.gemm_bf16(a, b, odd, a_mn, b_mn, None, 1.0, False, st, None)
    assert torch.equal(odd, guard[:M])
    assert int(st.item()) == 0


# 1, 128 rows and F = 264 (no 32-byte rows) are not served
@pytest.mark.parametrize("M,F,K", [(1, 64, 64), (128, 272, 128), (129, 16, 64), (300, 528, 200), (1500, 8960, 64), (200, 264, 64)])
def test_mlp_in(M, F, K):
    """Projections and activation in one launch: the bits of the plain GEMM followed by the elementwise kernel."""
    C, st = native(), status_word()
    torch.manual_seed(M + F)
    a = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device=DEV) * K ** -0.5).to(torch.bfloat16)
    act, alone, want = (torch.zeros(M, F, device=DEV, dtype=torch.bfloat16) for _ in range(3))
    gu, plain = (torch.zeros(M, 2 * F, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    served = C.gemm_mlp_in(a, w, act, gu, st)
    assert served == (M > 128 and F % 16 == 0) and C.gemm_mlp_in(a, w, alone, None, st) == served
    C.gemm_bf16(a, w, plain, False, False, None, 1.0, False, st, None)
    C.swiglu_fwd(plain, want)
    assert rel_err(plain.double(), a.double() @ w.double().t()) < BF16_TOL
    if served:
        assert torch.equal(gu, plain) and torch.equal(act, want) and torch.equal(alone, want)
    assert int(st.item()) == 0


@pytest.mark.parametrize("M,F", [(129, 16), (333, 528), (2100, 1040)])
def test_swiglu_with_row_scale(M, F):
    C, st = native(), status_word()
    torch.manual_seed(M)
    K = 256
    a = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device=DEV) * K ** -0.5).to(torch.bfloat16)
    ss = torch.round(a.double().pow(2).sum(1) * 2.0 ** 30).to(torch.int64)
    z = a.double() @ w.double().t() * torch.rsqrt(a.double().pow(2).mean(1, keepdim=True) + 1e-6)
    act = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
    C.gemm_swiglu(a, w, act, ss, 1e-6, st)
    assert int(st.item()) == 0
    assert rel_err(act.double(), torch.nn.functional.silu(z[:, :F]) * z[:, F:]) < BF16_TOL


@pytest.mark.parametrize("M,Hq,Hkv,K", [(129, 1, 1, 64), (300, 2, 1, 200), (777, 12, 2, 256), (128, 2, 1, 64)])
def test_qkv_with_rotation(M, Hq, Hkv, K):
    """The bits of the plain GEMM followed by the rotation kernel; a number of heads that ends inside a 256-wide tile, positions
    past the tables; 128 rows are not served."""
    C, st = native(), status_word()
    torch.manual_seed(M)
    N = (Hq + 2 * Hkv) * 128
    a = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = torch.randn(N, K, device=DEV).to(torch.bfloat16)
    bias = torch.randn(N, device=DEV).to(torch.bfloat16)
    pos = torch.randint(0, 500, (M,), device=DEV, dtype=torch.int32)
    ang = torch.randn(400, 64, device=DEV)
    cos_t, sin_t = ang.cos().contiguous(), ang.sin().contiguous()
    for b in (bias, None):
        got, want = (torch.zeros(M, N, device=DEV, dtype=torch.bfloat16) for _ in range(2))
        served = C.gemm_qkv_rope(a, w, got, b, pos, cos_t, sin_t, Hq + Hkv, 128, st)
        assert served == (M > 128)
        C.gemm_bf16(a, w, want, False, False, b, 1.0, False, st, None)
        C.rope_inplace(want, pos, cos_t, sin_t, Hq + Hkv, 128, False)
        if served:
            assert torch.equal(got, want)
    assert int(st.item()) == 0


# F = 264: no 32-byte rows; 128 rows: not served
# 6223 rows x 1536: 192-wide tiles
@pytest.mark.parametrize("M,F,K", [(129, 16, 64), (300, 528, 200), (1500, 8960, 64), (6223, 1536, 72), (128, 272, 64), (200, 264, 64)])
def test_swiglu_backward(M, F, K):
    """The bits of the plain GEMM followed by the elementwise kernel."""
    C, st = native(), status_word()
    torch.manual_seed(M + F)
    dy = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = torch.randn(K, F, device=DEV).to(torch.bfloat16)
    gu = (3 * torch.randn(M, 2 * F, device=DEV)).to(torch.bfloat16)
    gu[0, ::3], gu[0, 1::3] = 100.0, -100.0  # saturated gates
    got, want = (torch.zeros(M, 2 * F, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    dact = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
    served = C.gemm_swiglu_bwd(dy, w, gu, got, st)
    assert served == (M > 128 and F % 16 == 0)
    C.gemm_bf16(dy, w, dact, False, True, None, 1.0, False, st, None)
    C.swiglu_bwd(gu, dact, want)
    if served:
        assert torch.equal(got, want)
    assert int(st.item()) == 0
