"""A decoder layer as one native call against the same kernels called one by one, bit for bit; the decoder over resident parameters
(one call per layer) and over parameters handed out unit by unit (kernels called one by one)."""
import numpy as np
import pytest
import torch

from gpu_util import make_tiles, native, status_word

pytestmark = pytest.mark.gpu
DEV, EPS = "cuda", 1e-6
H, HQ, HKV, F = 512, 4, 2, 528


class Layer:
    """Flat parameters of one layer and the inputs of a packed batch; sequences of one tile, so that no sum depends on an order."""

    def __init__(self, lens, D=128, bias=True, seed=0):
        g = torch.Generator(device=DEV).manual_seed(seed)
        self.lens, self.D, self.T = lens, D, sum(lens)
        qd, cols = HQ * D, (HQ + 2 * HKV) * D
        shapes = dict(ln1=(H,), wqkv=(cols, H), bqkv=(cols,), wo=(H, qd), ln2=(H,), wgu=(2 * F, H), wd=(H, F))
        if not bias:
            del shapes["bqkv"]
        self.offs, n = {}, 0
        for k, s in shapes.items():
            self.offs[k] = n
            n += (torch.Size(s).numel() + 63) // 64 * 64
        self.shapes = shapes
        self.params = (torch.randn(n, device=DEV, generator=g) * 0.05).to(torch.bfloat16)
        for k in ("ln1", "ln2"):
            self.view(k).add_(1.0)
        self.grads = torch.randn(n, device=DEV, generator=g)
        self.x, self.dy = (torch.randn(self.T, H, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
        self.pos = torch.cat([torch.arange(m, dtype=torch.int32) for m in lens]).to(DEV)
        ang = torch.randn(128, D // 2, device=DEV, generator=g)
        self.cos, self.sin = ang.cos().contiguous(), ang.sin().contiguous()
        self.tiles, self.st = make_tiles(lens), status_word()
        self.dims = [H, HQ, HKV, D, F]
        self.off_list = [self.offs.get(k, -1) for k in ("ln1", "wqkv", "bqkv", "wo", "ln2", "wgu", "wd")]

    def view(self, k, flat=None):
        flat = self.params if flat is None else flat
        return flat[self.offs[k]:self.offs[k] + torch.Size(self.shapes[k]).numel()].view(self.shapes[k])

    def new(self, *shape, dtype=torch.bfloat16):
        return torch.zeros(shape, device=DEV, dtype=dtype)

    def gemm(self, a, b, out, a_mn=False, b_mn=False, bias=None, accumulate=False, residual=None):
        native().gemm_bf16(a, b, out, a_mn, b_mn, bias, 1.0, accumulate, self.st, residual)
        return out

    def forward(self):
        C, T, D = native(), self.T, self.D
        w, s = self.view, dict(rstd1=self.new(T, dtype=torch.float32), rstd2=self.new(T, dtype=torch.float32))
        s["h1"] = self.new(T, H)
        C.rmsnorm_fwd(self.x, w("ln1"), s["h1"], s["rstd1"], EPS)
        s["qkv"] = self.gemm(s["h1"], w("wqkv"), self.new(T, (HQ + 2 * HKV) * D), bias=w("bqkv") if "bqkv" in self.offs else None)
        C.rope_inplace(s["qkv"], self.pos, self.cos, self.sin, HQ + HKV, D, False)
        s["attn"], s["lse"] = self.new(T, HQ * D), self.new(HQ, T, dtype=torch.float32)
        C.attn_varlen_fwd(s["qkv"], s["attn"], s["lse"], self.tiles, HQ, HKV, D, D ** -0.5, self.st)
        s["x1"] = self.gemm(s["attn"], w("wo"), self.new(T, H), residual=self.x)
        s["h2"] = self.new(T, H)
        C.rmsnorm_fwd(s["x1"], w("ln2"), s["h2"], s["rstd2"], EPS)
        s["gu"], s["act"] = self.gemm(s["h2"], w("wgu"), self.new(T, 2 * F)), self.new(T, F)
        C.swiglu_fwd(s["gu"], s["act"])
        return self.gemm(s["act"], w("wd"), self.new(T, H), residual=s["x1"]), s

    def backward(self, s, grads):
        C, T, D = native(), self.T, self.D
        w, g, dx = self.view, lambda k: self.view(k, grads), self.dy.clone()
        dact, dgu = self.gemm(dx, w("wd"), self.new(T, F), b_mn=True), self.new(T, 2 * F)
        C.swiglu_bwd(s["gu"], dact, dgu)
        self.gemm(dx, s["act"], g("wd"), True, True, accumulate=True)
        dh = self.gemm(dgu, w("wgu"), self.new(T, H), b_mn=True)
        self.gemm(dgu, s["h2"], g("wgu"), True, True, accumulate=True)
        C.rmsnorm_bwd(dh, s["x1"], w("ln2"), s["rstd2"], dx, g("ln2"), True)
        dattn = self.gemm(dx, w("wo"), self.new(T, HQ * D), b_mn=True)
        self.gemm(dx, s["attn"], g("wo"), True, True, accumulate=True)
        dqkv, delta, acc = self.new(T, (HQ + 2 * HKV) * D), self.new(HQ, T, dtype=torch.float32), self.new(T, HQ * D, dtype=torch.float32)
        C.attn_varlen_bwd(s["qkv"], s["attn"], dattn, s["lse"], delta, acc, dqkv, self.tiles, HQ, HKV, D, D ** -0.5, self.st, self.pos, self.cos, self.sin)
        if "bqkv" in self.offs:
            C.colsum(dqkv, g("bqkv"))
        self.gemm(dqkv, w("wqkv"), dh, b_mn=True)
        self.gemm(dqkv, s["h1"], g("wqkv"), True, True, accumulate=True)
        C.rmsnorm_bwd(dh, self.x, w("ln1"), s["rstd1"], dx, g("ln1"), True)
        return dx

    def call_forward(self, keep, **kw):
        return native().layer_fwd(self.params, self.off_list, self.dims, EPS, self.x, self.pos, self.tiles, self.cos, self.sin, self.st, keep, **kw)

    def call_backward(self, slab, grads):
        dx = self.dy.clone()
        n = native().layer_bwd(self.params, grads, self.off_list, self.dims, EPS, dx, self.x, slab, self.pos, self.tiles, self.cos, self.sin, self.st)
        return dx, n


# one tile of rows; 129 - 256 rows: products with K-major operands are cut along K; more: CTA pairs. Heads of 64 are not rotated in the product
@pytest.mark.parametrize("lens", [[60], [100, 29], [128, 72], [128, 128], [128, 128, 44]])
@pytest.mark.parametrize("D,bias", [(128, True), (64, False)])
def test_layer_call(lens, D, bias):
    L = Layer(lens, D, bias, seed=sum(lens))
    want, s = L.forward()
    got, slab, _ = L.call_forward(True)
    assert torch.equal(got, want)
    assert torch.equal(L.call_forward(False)[0], want)
    g0, g1 = L.grads.clone(), L.grads.clone()
    want_dx = L.backward(s, g0)
    dx, _ = L.call_backward(slab, g1)
    assert int(L.st.item()) == 0
    assert torch.equal(dx, want_dx)
    for k in L.shapes:
        assert torch.equal(L.view(k, g1), L.view(k, g0)), k


class Units:
    """A provider of parameters unit by unit that has all of them at hand."""

    def __init__(self, layout, flat):
        self.layout, self.flat, self.device, self.status = layout, flat, flat.device, None

    def view(self, name):
        return self.layout.view(self.flat, name)

    def enter(self, unit, then):
        return 0

    def wants_ride(self, a, b):
        return False


def decoders(lens):
    from async_grpo_nccl_b200.models.config import PRESETS
    from async_grpo_nccl_b200.models.decoder import NativeDecoder
    from async_grpo_nccl_b200.models.layout import ParamLayout
    from async_grpo_nccl_b200.packing import pack_samples

    cfg = PRESETS["tiny128"]
    layout = ParamLayout(cfg)
    p32 = torch.empty(layout.total)
    layout.init_random_(p32, 0)
    flat = p32.to(torch.bfloat16).to(DEV)
    rng = np.random.default_rng(3)
    samples = [{"sample_ids": rng.integers(0, cfg.vocab_size, n).astype(np.int32), "input_len": n // 3, "output_len": n - n // 3, "advantage": 1.0}
               for n in lens]
    batch = pack_samples(samples, pin=False).to_device(DEV)
    return cfg, layout, batch, NativeDecoder(cfg, layout, flat), NativeDecoder(cfg, layout, None, weights=Units(layout, flat))


def test_prompt_layer_writes_the_cache_with_either_kind_of_parameters():
    cfg, layout, batch, resident, sharded = decoders([40, 100, 7])
    T, bs = batch.T, 16
    blocks = (T + bs - 1) // bs
    slots = torch.randperm(blocks * bs, generator=torch.Generator().manual_seed(0))[:T].to(torch.int32).to(DEV)
    x = torch.randn(T, cfg.hidden_size, device=DEV).to(torch.bfloat16)
    got = []
    for dec in (resident, sharded):
        k, v = (torch.full((blocks, cfg.num_key_value_heads, bs, cfg.head_dim), 5.0, device=DEV, dtype=torch.bfloat16) for _ in range(2))
        cos_t, sin_t = dec.rope_tables(1)
        out = dec._layer_fwd(0, x, batch, cos_t, sin_t, None, kv_write=(k, v, slots))
        dec.check_status()
        got.append((out, k, v))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    assert int((got[1][1] != 5.0).any(-1).any(1).sum()) == T


def package_kernels(fn):
    """Kernels of this package that `fn` launches."""
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    return sum(e.count for e in p.key_averages() if "agrpo" in e.key)


# 60 rows: plain kernels; 200: products cut along K; 400: CTA pairs
@pytest.mark.parametrize("lens", [[60], [120, 80], [128, 128, 144]])
def test_launches_are_counted(lens):
    from async_grpo_nccl_b200.models.decoder import GradSink, LossConfig

    cfg, layout, batch, resident, sharded = decoders(lens)
    lc, sink = LossConfig(kl_beta=0.0, temperature=1.0), GradSink(layout, DEV)
    for dec in (resident, sharded):
        for fn in (lambda: dec.logprobs(batch, 1.0), lambda: dec.forward_backward(batch, lc, 0.5, sink)):
            fn()
            before = dec.launches
            seen = package_kernels(fn)
            assert dec.launches - before == seen
