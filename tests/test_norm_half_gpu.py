"""The staged norms in fp16: every number of warps to a row, forward and backward, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer", [True, False])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 264), (301, 768), (700, 1024), (500, 1032), (300, 1544), (777, 3072), (90, 3080)])
@pytest.mark.parametrize("res", [True, False])
def test_half_against_64_bits(rows, cols, layer, res):
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(rows + cols)
    x, r, dy, dres = (torch.randn(rows, cols, device="cuda").half() for _ in range(4))
    w = (torch.randn(cols, device="cuda") * 0.2 + 1.0).half()
    b = torch.randn(cols, device="cuda").half() if layer else None
    y, h, rstd, mean = E.norm_fwd(x, w, b, r if res else None, eps=1e-5, layer=layer)
    assert torch.equal(h, (x.float() + r.float()).half() if res else x)
    hd, wd, gd = h.double(), w.double(), dy.double()
    mu = hd.mean(1, keepdim=True) if layer else torch.zeros(rows, 1, device="cuda", dtype=torch.float64)
    rs = ((hd - mu).pow(2).mean(1, keepdim=True) + 1e-5).rsqrt()
    xh = (hd - mu) * rs
    want = xh * wd + (b.double() if layer else 0.0)
    # one rounding to fp16 of a result whose terms (the value and the bias) carry a few units of fp32
    assert ((y.double() - want).abs() <= want.abs() * 2.0 ** -11 + 1e-5).all()
    assert ((rstd.double() - rs[:, 0]).abs() <= 1e-5 * rs[:, 0]).all()
    dh, dw, db = E.norm_bwd(dy, h, w, rstd, mean, dres if res else None, layer=layer, has_bias=layer)
    assert E.norm_error() == 0
    gw = gd * wd
    want = rs * (gw - xh * (gw * xh).mean(1, keepdim=True) - (gw.mean(1, keepdim=True) if layer else 0.0)) + (dres.double() if res else 0.0)
    # as the bf16 form of test_norm_bwd_gpu.py, with the rounding of fp16; the column sums are rounded to it as well
    assert ((dh.double() - want).abs() <= want.abs() * 2.0 ** -11 + 2e-5 * gw.abs().amax(1, keepdim=True) * rs).all()
    tol = 1e-6 * rows ** 0.5 * 40 + 1e-6
    sums = [(dw, (gd * xh).sum(0))] + ([(db, gd.sum(0))] if layer else [])
    for got, ref in sums:
        assert ((got.double() - ref).abs() <= ref.abs() * 2.0 ** -11 + tol).all()
