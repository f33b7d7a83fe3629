"""The persistent decode kernel's hand-off by value: more splits than heads, than tokens and than one pass merges, page numbers beyond
the first 32 blocks a warp, newest tokens at block edges, sums that are not finite; what it leaves behind in its buffers."""
import math

import pytest
import torch

from gpu_util import native, rel_err, status_word
from test_decode_layers_gpu import _reference

pytestmark = pytest.mark.gpu
DEV, D, BS, EPS = "cuda", 128, 16, 1e-6


class Case:
    def __init__(self, lens, splits, H=512, Hq=4, Hkv=2, F=1408, L=2):
        torch.manual_seed(len(lens) + splits)
        self.B, self.splits, self.H, self.Hq, self.Hkv, self.F, self.L = len(lens), splits, H, Hq, Hkv, F, L
        B, Q, QD = self.B, (Hq + 2 * Hkv) * D, Hq * D
        w = lambda *s: (torch.randn(*s, device=DEV) * (0.5 / math.sqrt(s[-1]))).to(torch.bfloat16)
        self.Wq, self.Wo, self.Wgu, self.Wd = w(L, Q, H), w(L, H, QD), w(L, 2 * F, H), w(L, H, F)
        self.bq = (torch.randn(L, Q, device=DEV) * 0.1).to(torch.bfloat16)
        self.lens = torch.tensor(lens, device=DEV, dtype=torch.int32)
        blocks = [(n + BS - 1) // BS for n in lens]
        self.cache = (torch.randn(L, 2, sum(blocks) + 3, Hkv, BS, D, device=DEV) * 0.5).to(torch.bfloat16)
        perm = torch.randperm(sum(blocks) + 3, device=DEV).to(torch.int32)
        self.bt = torch.full((B, max(blocks)), -1, device=DEV, dtype=torch.int32)
        at = 0
        for b, n in enumerate(blocks):
            self.bt[b, :n] = perm[at:at + n]
            at += n
        ang = torch.arange(max(lens) + 1, device=DEV).float()[:, None] / (10000.0 ** (torch.arange(0, D, 2, device=DEV).float() / D))
        self.cos, self.sin = ang.cos().contiguous(), ang.sin().contiguous()
        self.x0 = torch.randn(B, H, device=DEV).to(torch.bfloat16)
        C = native()
        self.rows = 32 if B <= 32 else 64
        new = lambda n: torch.zeros(self.rows, n, device=DEV, dtype=torch.bfloat16)
        self.x, self.x1, self.qkv, self.attn, self.act = new(H), new(H), new(Q), new(QD), new(F)
        self.ss = torch.zeros(2 * L + 1, self.rows, device=DEV, dtype=torch.int64)
        self.part_o, self.part_ml = torch.zeros(B * Hkv * splits * 8 * D, device=DEV), torch.zeros(B * Hkv * splits * 16, device=DEV)
        self.tickets = torch.zeros(B * Hkv, device=DEV, dtype=torch.int32)
        self.partials = torch.zeros(C.decode_layers_scratch_bytes(B, H, Q, QD, F) // 4, device=DEV)
        self.counters = torch.zeros(C.decode_layers_counter_words(), device=DEV, dtype=torch.int32)

    def run(self, x0, with_status=True):
        C, st = native(), status_word() if with_status else None
        self.x[:self.B] = x0
        self.ss.zero_()
        self.ss[0, :self.B] = ((x0.nan_to_num(0, 0, 0).double() ** 2).sum(-1) * 2 ** 30).round().to(torch.int64)
        cache = self.cache.clone()
        s = lambda t: t[0].numel()
        C.decode_layers(self.L, self.B, self.Wq[0], s(self.Wq), self.Wo[0], s(self.Wo), self.Wgu[0], s(self.Wgu), self.Wd[0], s(self.Wd), self.bq[0],
                        s(self.bq), self.x, self.x1, self.qkv, self.attn, self.act, self.ss, EPS, self.cos, self.sin, self.bt, self.lens, cache,
                        self.Hq, self.Hkv, 1 / math.sqrt(D), self.splits, self.part_o, self.part_ml, self.tickets, self.partials, self.counters, st)
        torch.cuda.synchronize()
        assert st is None or int(st.item()) == 0
        return self.x[:self.B].clone(), cache

    def check_left_behind(self):
        """Every word that was handed over reads "not yet" again: the launch sets the buffers so, a reader puts it back."""
        for t in (self.partials, self.part_o, self.part_ml)[:3 if self.splits > 1 else 1]:
            assert bool((t.view(torch.int32) == -1).all())


@pytest.mark.parametrize("lens,splits", [
    ([1, 16, 17, 700], 8),               # fewer heads a group (2) than splits; splits without a block
    ([1, 15, 33, 2049, 64], 12),         # merged in two passes
    ([5, 16, 400], 9),
    ([2049, 4200, 1, 17, 2048], 1),      # more than 32 blocks a warp
    ([4600] + [33] * 32, 3),             # a row tile of 64
])
def test_splits_and_block_edges(lens, splits):
    c = Case(lens, splits)
    ref_x, ref_k, ref_v = _reference(c.x0, c.Wq, c.Wo, c.Wgu, c.Wd, c.bq, c.cache, c.bt, c.lens, c.cos, c.sin, c.Hq, c.Hkv, EPS)
    x, cache = c.run(c.x0)
    c.check_left_behind()
    assert rel_err(x, ref_x) < 3e-2
    assert rel_err(cache[:, 0], ref_k.float()) < 2e-2 and rel_err(cache[:, 1], ref_v.float()) < 2e-2
    again, _ = c.run(c.x0, with_status=False)
    assert torch.equal(again, x)


# A row of NaN (every payload is one the kernel may meet, the reserved pattern's bf16 half among them), of infinities, of both: the launch
# ends, the other rows have the bits that they have without it.
@pytest.mark.parametrize("bits", [0x7fc0, 0xffff, 0x7f80, 0xff80])
@pytest.mark.parametrize("splits", [1, 3])
def test_sums_that_are_not_finite(bits, splits):
    c = Case([40, 300, 17, 129, 64], splits)
    want, _ = c.run(c.x0)
    assert bool(torch.isfinite(want).all())
    x0 = c.x0.clone()
    x0.view(torch.int16)[2] = bits - (1 << 16) if bits >= 1 << 15 else bits
    got, _ = c.run(x0)
    c.check_left_behind()
    rest = [0, 1, 3, 4]
    assert torch.equal(got[rest], want[rest])
    assert not bool(torch.isfinite(got[2].float()).any())
    again, _ = c.run(c.x0)
    assert torch.equal(again, want)
