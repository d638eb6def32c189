"""AdamW with state on 32-byte boundaries (one access per eight values) and off them (two): the same bits, ragged ends included."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [1, 7, 8, 4095, 4096, 4104, 65536 + 4096 + 5])
def test_alignment_of_the_state_does_not_matter(n, dtype):
    from zen_repro_b200.optim.adamw import FusedAdamW

    gen = torch.Generator("cuda").manual_seed(n)
    start = torch.randn(n, device="cuda", generator=gen).to(dtype)
    grads = [torch.randn(n, device="cuda", generator=gen).to(dtype) for _ in range(3)]

    def run(off):
        p = torch.nn.Parameter(start.clone())
        opt = FusedAdamW([p], lr=1e-3)
        st = opt._init_state(p)
        for k in ("exp_avg", "exp_avg_sq", "master"):
            if k in st:
                buf = torch.empty(n + off, dtype=torch.float32, device="cuda")
                buf[off:] = st[k]
                st[k] = buf[off:]
        for g in grads:
            p.grad = g.clone()
            opt.step(clear_grads=True)
        assert int((p.grad != 0).sum()) == 0
        return [p.detach(), st["exp_avg"], st["exp_avg_sq"]]

    for a, b in zip(run(0), run(4)):
        assert torch.equal(a, b)
