"""The library's own count of its launches against the kernels that a profiler sees on the device."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CONFIGS = {
    "gpt2": dict(hidden_size=128, num_heads=2, num_kv_heads=2, head_dim=64, intermediate_size=512),
    "google/gemma-2-2b": dict(hidden_size=128, num_heads=4, num_kv_heads=1, head_dim=256, intermediate_size=256),
}


def _own_kernels(run):
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    library = ("at::", "cub::", "cublas", "cutlass", "nvjet", "Memcpy", "Memset")
    return [n for n in names if not any(k in n for k in library)]


@pytest.mark.parametrize("name,bsz,seq", [("gpt2", 2, 64), ("gpt2", 1, 700), ("google/gemma-2-2b", 1, 300)])
@pytest.mark.parametrize("train", [True, False])
def test_model_pass(name, bsz, seq, train):
    from zen_repro_b200 import _native
    from zen_repro_b200.models import build_model

    model = build_model(name, device="cuda", num_layers=2, vocab_size=512, max_position=1024, **CONFIGS[name])
    ids = torch.randint(0, 512, (bsz, seq), device="cuda")

    def step():
        with torch.set_grad_enabled(train):
            loss = model(ids, ids)
        if train:
            loss.backward()

    step()
    before = _native.launch_count()
    own = _own_kernels(step)
    assert _native.launch_count() - before == len(own) > 10, own


@pytest.mark.parametrize("method", [1, 3])
def test_sparse_call(method):
    from zen_repro_b200 import _native
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    eng = VirtualSparseAllReduce(10_000, 3, max_density=0.2, methods=(method,))
    xs = [torch.where(torch.rand(10_000, device="cuda") < 0.05, 1.0, 0.0) for _ in range(3)]
    eng(xs, method=method)
    before = _native.launch_count()
    own = _own_kernels(lambda: eng(xs, method=method))
    assert _native.launch_count() - before == len(own) == 4, own
