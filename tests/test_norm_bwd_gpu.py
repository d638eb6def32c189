"""Norm backward in one pass: every number of warps to a row, rows that do not fill a stage or a chunk, with and without the residual
gradient, and the column sums of the result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer", [True, False])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 264), (64, 768), (301, 768), (5000, 1024), (2500, 1032), (900, 2304), (777, 3072), (600, 3080), (40, 8192), (9999, 256),
                                       (500, 776), (300, 1544)])
def test_against_64_bits(rows, cols, layer):
    from zen_repro_b200 import _native

    lib = _native.lib()
    torch.manual_seed(rows + cols)
    dy, h, dres = (torch.randn(rows, cols, device="cuda").bfloat16() for _ in range(3))
    w = (torch.randn(cols, device="cuda") * 0.2 + 1.0).bfloat16()
    hd = h.double()
    mean = hd.mean(1) if layer else torch.zeros(rows, device="cuda", dtype=torch.float64)
    rstd = ((hd - mean[:, None]).pow(2).mean(1) + 1e-5).rsqrt()
    xh = (hd - mean[:, None]) * rstd[:, None]
    gw = dy.double() * w.double()
    t = gw - xh * (gw * xh).mean(1, keepdim=True) - (gw.mean(1, keepdim=True) if layer else 0.0)
    base = rstd[:, None] * t
    parts = lib.zen_norm_bwd_parts_used(rows, cols)
    fm, fr = mean.float(), rstd.float()
    for res, sums in ((True, True), (True, False), (False, True), (False, False)):
        dh = torch.empty_like(h)
        pw, pb, ph = (torch.full((parts, cols), float("nan"), device="cuda") for _ in range(3))
        rc = lib.zen_norm_bwd_sums(dy.data_ptr(), h.data_ptr(), w.data_ptr(), fr.data_ptr(), fm.data_ptr() if layer else 0, dres.data_ptr() if res else 0,
                                   dh.data_ptr(), pw.data_ptr(), pb.data_ptr() if layer else 0, ph.data_ptr() if sums else 0, 0, 0, rows, cols, int(layer), 0,
                                   0, 1, 1, _native.stream_ptr())
        assert rc == 0 and lib.zen_norm_error() == 0
        want = base + (dres.double() if res else 0.0)
        # one rounding to bf16; fp32 sums of a row are off by a few units of its largest term
        assert ((dh.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5 * gw.abs().amax(1, keepdim=True) * rstd[:, None]).all()
        tol = 1e-6 * rows ** 0.5 * 40 + 1e-6
        assert ((pw.double().sum(0) - (dy.double() * xh).sum(0)).abs() <= tol).all()
        if layer:
            assert ((pb.double().sum(0) - dy.double().sum(0)).abs() <= tol).all()
        if sums:
            assert ((ph.double().sum(0) - dh.double().sum(0)).abs() <= tol * (1 + float(dh.abs().max()))).all()


@pytest.mark.parametrize("layer", [True, False])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 264), (64, 768), (301, 768), (5000, 1024), (2500, 1032), (900, 2304), (777, 3072), (600, 3080), (9999, 256), (500, 776),
                                       (300, 1544)])
def test_forward_against_64_bits(rows, cols, layer):
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(rows * 3 + cols)
    x, res = (torch.randn(rows, cols, device="cuda").bfloat16() for _ in range(2))
    w = (torch.randn(cols, device="cuda") * 0.2 + 1.0).bfloat16()
    b = torch.randn(cols, device="cuda").bfloat16() if layer else None
    for r in (res, None):
        y, h, rstd, mean = E.norm_fwd(x, w, b, r, eps=1e-5, layer=layer)
        assert E.norm_error() == 0
        want_h = (x.float() + r.float()).bfloat16() if r is not None else x
        assert torch.equal(h, want_h)
        hd = want_h.double()
        mu = hd.mean(1, keepdim=True) if layer else 0.0
        rs = ((hd - mu).pow(2).mean(1, keepdim=True) + 1e-5).rsqrt()
        want = (hd - mu) * rs * w.double() + (b.double() if layer else 0.0)
        # one rounding to bf16 of a result whose terms (the value and the bias) carry a few units of fp32
        assert ((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()
        assert ((rstd.double() - rs[:, 0]).abs() <= 1e-5 * rs[:, 0]).all()
        if layer:
            assert ((mean.double() - mu[:, 0]).abs() <= 1e-6).all()
