"""RMSNorm backward where its grid and the sum of the parked shares of dW change: rows around the number of CTAs (two
or four per SM) and around 128, the partials requested together; narrow and wide rows.  Against float64: dX and dW
are rounded once to 16 bits (2^-9 relative in bf16); dW also carries fp32 sums of `rows` products."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 7, 127, 128, 129, 295, 297, 591, 592, 593, 1300])
@pytest.mark.parametrize("cols", [8, 1000, 2048, 2056, 4096, 4104])
def test_backward_at_the_edges_of_grid_and_partials(dtype, rows, cols):
    from loquetier_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    x = (torch.randn((rows, cols), generator=g, device=DEV) * 1.5).to(dtype)
    go = torch.randn((rows, cols), generator=g, device=DEV).to(dtype)
    w = (1.0 + 0.1 * torch.randn(cols, generator=g, device=DEV)).to(dtype)
    out, rms = torch.empty_like(x), torch.empty((rows, 1), dtype=torch.float32, device=DEV)
    ops.rms_norm(out, rms, x, w, 1e-5)
    dx, dw = torch.full_like(x, float("nan")), torch.full((cols,), float("nan"), dtype=torch.float32, device=DEV)
    ops.rms_norm_bwd(dx, dw, go, x, w, rms)
    xd, gd, wd = x.double(), go.double(), w.double()
    s = torch.rsqrt((xd * xd).mean(1, keepdim=True) + 1e-5)
    want_dw = (xd * s * gd).sum(0)
    want_dx = (gd * wd - xd * (gd * wd * xd).mean(1, keepdim=True) * s * s) * s
    assert ((dx.double() - want_dx).abs() <= 2 ** -8 * want_dx.abs() + 1e-4).all()
    assert ((dw.double() - want_dw).abs() <= 1e-5 * rows ** 0.5 * (1 + want_dw.abs())).all()
    dw2 = torch.empty_like(dw)
    ops.rms_norm_bwd(dx, dw2, go, x, w, rms)
    assert torch.equal(dw, dw2)   # added in a fixed order
