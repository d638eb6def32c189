"""Activations at sizes that end inside a thread's group of vectors, one row, one vector, the halves of one matrix, every mode."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("rows,inner", [(0, 8), (1, 8), (3, 520), (257, 64), (1000, 3080), (5, 16384)])
def test_forward_and_backward(rows, inner, mode):
    from zen_repro_b200 import _native

    lib, st = _native.lib(), _native.stream_ptr()
    torch.manual_seed(rows + inner)
    w = 2 if mode >= 2 else 1
    u = torch.randn(rows, inner * w, device="cuda").bfloat16()
    dm = torch.randn(rows, inner, device="cuda").bfloat16()
    m, du = torch.full_like(dm, 9.0), torch.full_like(u, 9.0)
    half = inner * 2
    assert lib.zen_act_fwd(u.data_ptr(), u.data_ptr() + half, m.data_ptr(), rows, inner, inner * w, inner * w, mode, 1, st) == 0
    assert lib.zen_act_bwd(u.data_ptr(), u.data_ptr() + half, dm.data_ptr(), du.data_ptr(), du.data_ptr() + half, rows, inner, inner * w, inner * w, mode, 1,
                           st) == 0
    x = u.float().requires_grad_(True)
    a, b = (x[:, :inner], x[:, inner:]) if w == 2 else (x, None)
    want = [lambda: F.gelu(a, approximate="tanh"), lambda: F.relu(a), lambda: F.silu(a) * b, lambda: F.gelu(a, approximate="tanh") * b][mode]()
    (g,) = torch.autograd.grad(want, x, dm.float())
    # tanh.approx is good to 2^-11, the result to 2^-9
    torch.testing.assert_close(m.float(), want.detach(), atol=4e-3, rtol=1e-2)
    torch.testing.assert_close(du.float(), g, atol=1e-2, rtol=1e-2)
