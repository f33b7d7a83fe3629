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
