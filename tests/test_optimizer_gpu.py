"""The AdamW kernel: sizes that are no multiple of four and buffers that no 16-byte access fits, against fp64."""
import pytest
import torch

from gpu_util import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (4096, 0), (1001, 0), (1000, 1)])
def test_adamw_sizes(n, off):
    C = native()
    torch.manual_seed(n)
    g, p, m, v = (torch.randn(n + off, device="cuda")[off:] for _ in range(4))
    v.abs_()
    p16 = torch.empty(n + off, device="cuda", dtype=torch.bfloat16)[off:]
    norm = g.double().pow(2).sum().float().reshape(1)
    lr, b1, b2, eps, wd, step = 1e-2, 0.9, 0.95, 1e-8, 0.1, 3
    gd = g.double() * min(1.0, 1.0 / (float(norm.sqrt()) + 1e-6))
    md, vd = b1 * m.double() + (1 - b1) * gd, b2 * v.double() + (1 - b2) * gd * gd
    want = p.double() * (1 - lr * wd) - lr / (1 - b1 ** step) * md / ((vd / (1 - b2 ** step)).sqrt() + eps)
    C.adamw_step(p, m, v, g, p16, lr, b1, b2, eps, wd, step, 1.0, norm, 1.0, True)
    # a dozen fp32 roundings and the fast square root and division (2 ulp each); the step is at most a few lr = 0.01 wide
    tol = 32 * 2.0 ** -24
    for got, ref in ((m, md), (v, vd), (p, want)):
        assert ((got.double() - ref).abs() <= tol * (ref.abs() + 1)).all()
    assert torch.equal(p16, p.to(torch.bfloat16)) and not g.any()


# Buffers of 16-byte alignment (each its own), sizes around a multiple of four and eight, against aligned ones: the same operations, which
# the compiler may contract differently in the loop for the rest.
@pytest.mark.parametrize("n,off", [(1, (4, 4, 4, 4, 4)), (3, (4, 0, 4, 4, 0)), (4, (4, 4, 4, 4, 4)), (8191, (4, 8, 12, 0, 4)), (40000, (0, 0, 0, 0, 4))])
def test_adamw_slices_of_16_bytes(n, off):
    C = native()
    torch.manual_seed(n)
    src = [torch.randn(n, device="cuda") for _ in range(4)]
    src[2].abs_()
    results = []
    for offs in ((0,) * 5, off):
        bufs = [torch.cat([torch.full((o,), 7.0, device="cuda"), t, torch.full((9,), 7.0, device="cuda")]) for o, t in zip(offs, src)]
        p, m, v, g = (b[o:o + n] for o, b in zip(offs, bufs))
        b16 = torch.full((n + offs[4] + 9,), 7.0, device="cuda", dtype=torch.bfloat16)
        p16 = b16[offs[4]:offs[4] + n]
        C.adamw_step(p, m, v, g, p16, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, 1.0, torch.ones(1, device="cuda"), 1.0, True)
        for o, b in zip(offs, bufs + [b16]):
            assert (b[:o] == 7).all() and (b[o + n:] == 7).all()
        results.append([t.clone() for t in (p, m, v)])
        assert torch.equal(p16, p.to(torch.bfloat16)) and not g.any()
    assert all(((a - b).abs() <= 32 * 2.0 ** -24 * (b.abs() + 1)).all() for a, b in zip(*results))


def test_adamw_slice_of_16_bytes_keeps_wide_accesses():
    C = native()
    n = 64 << 20
    times = []
    for off in (0, 4):
        p, m, v, g = (torch.zeros(n + off, device="cuda")[off:] for _ in range(4))
        p16 = torch.zeros(n + off, device="cuda", dtype=torch.bfloat16)[off:]
        run = lambda: C.adamw_step(p, m, v, g, p16, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, 1.0, torch.ones(1, device="cuda"), 1.0, True)
        for _ in range(3):
            run()
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(11)]
        for e in ev[:-1]:
            e.record()
            run()
        ev[-1].record()
        torch.cuda.synchronize()
        times.append(sorted(a.elapsed_time(b) for a, b in zip(ev, ev[1:]))[5])
    assert times[1] < 1.5 * times[0], times  # 0.341 and 0.346 ms; 0.683 with one parameter a thread
