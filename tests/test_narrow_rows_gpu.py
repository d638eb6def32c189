"""Rows beyond the last whole 256 as transposed tiles of the CTA-pair GEMM: every edge of such a tile, both layouts of B, with a bias."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows over: 1 (the second CTA's rows all beyond the matrix), 32 and 33 (widths 32 and 64), 44, 128 (the widest); columns: whole tiles, a
# remainder, an odd number in a wider buffer; depth: one block of K, a remainder of one, more blocks than stages.  The last two keep whole
# tiles: 129 rows over, and too few rounds.
@pytest.mark.parametrize("m,n,k", [(257, 16384, 64), (288, 50000, 200), (289, 50008, 1024), (300, 50257, 456), (777, 128256, 1024), (384, 128256, 64),
                                   (1290, 16384, 128), (1300, 16384, 960), (385, 128256, 64), (2100, 2304, 768)])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("bias", [False, True])
def test_rows_beyond_the_last_whole_tile(m, n, k, b_mn, bias):
    from zen_repro_b200 import _native
    from zen_repro_b200.ops import gemm as G

    if b_mn and n % 8:
        pytest.skip("rows of such a B are not aligned: copied, and the same as aligned ones from there on")
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn(n, k, device="cuda").bfloat16()
    v = torch.randn(n, device="cuda").bfloat16() if bias else None
    ld = (n + 7) // 8 * 8

    def run():
        buf = torch.full((m + 3, ld + 8), 7.0, dtype=torch.bfloat16, device="cuda")
        out = buf[:m, :n]
        if b_mn:
            bt = b.t().contiguous()
            G._launch(a, bt, m, n, k, False, True, v, out, False, None, 512, last=True)
        else:
            G.gemm_nt(a, b, bias=v, out=out, bn=512, pad_ok=True, last=True)
        assert (buf[m:] == 7.0).all() and (buf[:, ld:] == 7.0).all()     # nothing beyond the matrix and its padding
        assert b_mn or (buf[:m, n:ld] == 0.0).all()                      # which is written with zeros
        return out.float()

    got = run()
    old = _native.lib().zen_gemm2_tail_split(0)
    try:
        whole = run()
    finally:
        _native.lib().zen_gemm2_tail_split(old)
    assert torch.equal(got, whole)                                       # the same products in the same order
    rows = torch.tensor([0, 255, m // 256 * 256 - 1, m // 256 * 256, m - 1], device="cuda")
    ref = a[rows].double() @ b.double().t() + (v.double() if bias else 0.0)
    # one rounding to bf16 of a sum whose fp32 error is at most (k + 1) 2^-24 of the magnitudes added
    mag = a[rows].double().abs() @ b.double().abs().t() + (v.double().abs() if bias else 0.0)
    assert ((got[rows].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + mag * (k + 1) * 2.0 ** -23).all()
