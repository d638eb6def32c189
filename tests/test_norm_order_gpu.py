"""The statistics of a norm do not depend on the kernel that takes them: the staged kernel of the 16-bit types adds in the order of the
kernels that fp32 goes through, so that equal values give equal bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [8, 768, 776, 1024, 1032, 2048, 2304, 3072])
@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("rows", [1, 700])
def test_statistics_equal_those_of_fp32(cols, layer, rows):
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(cols + rows)
    x = (torch.randn(rows, cols, device="cuda") + 0.5).bfloat16()
    w, b = torch.randn(cols, device="cuda").bfloat16(), torch.randn(cols, device="cuda").bfloat16() if layer else None
    y, _, *stats = E.norm_fwd(x, w, b, eps=1e-5, layer=layer)
    y32, _, *stats32 = E.norm_fwd(x.float(), w.float(), b.float() if layer else None, eps=1e-5, layer=layer)
    assert E.norm_error() == 0
    for one, two in zip(stats, stats32):
        assert (one is None) == (two is None) and (one is None or torch.equal(one, two))
    assert torch.equal(y, y32.bfloat16())
