"""RMSNorm backward over many rows (``csrc/elementwise.cu``) against float64."""
import pytest
import torch

from adaptivetrainingsystem_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows: fewer than the groups of the grid, one more than a whole round of them, several rounds; columns around the widths of the groups
@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("rows,cols", [(1024, 8), (1190, 256), (1200, 264), (3111, 512), (1500, 520), (2369, 768), (1300, 776), (1185, 1000), (3000, 1024), (1184, 1032), (2000, 1536), (1500, 1544), (2500, 2048), (1030, 2056), (1777, 4096), (1024, 8192), (1100, 16384)])
def test_backward_of_many_rows(rows, cols, skip):
    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    x0, dy, ds = (torch.randn(rows, cols, generator=g, device=DEV).bfloat16() for _ in range(3))
    w0, eps = (1 + 0.1 * torch.randn(cols, generator=g, device=DEV)).bfloat16(), 1e-6
    x, w = x0.clone().requires_grad_(), w0.clone().requires_grad_()
    if skip:
        y, through = ops.rms_norm_skip(x, w, eps)
        torch.autograd.backward([y, through], [dy, ds])
    else:
        ops.rms_norm(x, w, eps).backward(dy)
    xd, wd, d = x0.double(), w0.double(), dy.double()
    r = torch.rsqrt((xd ** 2).mean(-1, keepdim=True) + eps)
    xh = xd * r
    want = r * (d * wd - xh * (d * wd * xh).mean(-1, keepdim=True)) + (ds.double() if skip else 0)
    # fp32 throughout (the two terms of a difference, a mean over the columns), one rounding to bf16
    mass = r * ((d * wd).abs() + xh.abs() * (d * wd * xh).abs().mean(-1, keepdim=True)) + (ds.double().abs() if skip else 0)
    assert bool(((x.grad.double() - want).abs() <= 2.0 ** -8 * want.abs() + 64 * 2.0 ** -23 * mass).all())
    dw, dmass = (d * xh).sum(0), (d * xh).abs().sum(0)
    assert bool(((w.grad.double() - dw).abs() <= 2.0 ** -8 * dw.abs() + (rows + 16) * 2.0 ** -23 * dmass).all())
