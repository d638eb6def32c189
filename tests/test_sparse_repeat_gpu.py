"""Many calls of a size whose stages are reused soon after they were read: every one exact (a stage that is overwritten while a lane still
reads it showed in one call of fifty)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,dtype", [(8, torch.bfloat16), (8, torch.float32), (4, torch.bfloat16), (3, torch.float16), (2, torch.float32)])
def test_repeated_calls_stay_exact(P, dtype):
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    n = 3_000_017
    eng = VirtualSparseAllReduce(n, P, max_density=0.065, methods=(3,), deterministic=True)
    gen = torch.Generator("cuda").manual_seed(1)
    xs = [torch.where(torch.rand(n, device="cuda", generator=gen) < 0.05, torch.randn(n, device="cuda", generator=gen),
                      torch.zeros((), device="cuda")).to(dtype) for _ in range(P)]
    want = torch.zeros(n, device="cuda")
    for x in xs:
        want += x.float()
    want = want.to(dtype)
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(400):
        outs = eng(xs, method=3)
        wrong += (outs[i % P] != want).any()
    assert eng.status() == [0] * P
    assert int(wrong) == 0
