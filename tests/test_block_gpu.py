"""The native decoder block against the op-by-op path: every family's layout, first block (no residual), ragged tokens,
gradients through autograd and straight into the reducer's buckets."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CONFIGS = {
    "gpt2": dict(hidden_size=128, num_heads=2, num_kv_heads=2, head_dim=64, intermediate_size=512),
    "facebook/opt-2.7b": dict(hidden_size=160, num_heads=2, num_kv_heads=2, head_dim=80, intermediate_size=640),
    "meta-llama/Llama-3.2-3B": dict(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=64, intermediate_size=320),
    "gemma-2b": dict(hidden_size=136, num_heads=4, num_kv_heads=1, head_dim=256, intermediate_size=264),
    "google/gemma-2-2b": dict(hidden_size=128, num_heads=2, num_kv_heads=1, head_dim=256, intermediate_size=256),
}


@pytest.mark.parametrize("name,bsz,seq", [("gpt2", 2, 64), ("gpt2", 1, 7), ("facebook/opt-2.7b", 3, 100), ("meta-llama/Llama-3.2-3B", 1, 333),
                                          ("gemma-2b", 2, 77), ("google/gemma-2-2b", 2, 128)])
@pytest.mark.parametrize("buckets", [False, True])
def test_matches_op_by_op(name, bsz, seq, buckets, monkeypatch):
    from zen_repro_b200.models import build_model
    from zen_repro_b200.ops import block
    from zen_repro_b200.parallel import ZenDDP

    model = build_model(name, device="cuda", num_layers=2, vocab_size=512, max_position=512, **CONFIGS[name])
    model.reset_parameters(seed=1)
    with torch.no_grad():
        for n, p in model.named_parameters():
            if n.endswith("_b"):
                p.normal_(0.0, 0.02)
    ids = torch.randint(0, 512, (bsz, seq), device="cuda")
    calls = []
    real = block.run
    monkeypatch.setattr(block, "run", lambda *a: calls.append(1) or real(*a))

    def step():
        m = ZenDDP(model) if buckets else model
        if not buckets:
            for p in model.parameters():
                p.grad = None
                p.zen_direct_grad = False
        loss = m(ids, ids)
        loss.backward()
        if buckets:
            m.finalize_grads()
        return loss.detach(), {n: p.grad.detach().clone() for n, p in model.named_parameters()}

    loss, grads = step()
    assert len(calls) == 2
    monkeypatch.setattr(block, "usable", lambda *a: False)
    want_loss, want = step()
    assert len(calls) == 2
    assert abs(float(loss - want_loss)) < 1e-3
    for n in want:
        assert (grads[n].float() - want[n].float()).norm() <= 1e-2 * want[n].float().norm() + 1e-7, n


def test_parameters_given_other_storage_before_the_backward():
    """The backward reads the weights where they are then, not where the forward found them."""
    from zen_repro_b200.models import build_model

    model = build_model("gpt2", device="cuda", num_layers=2, vocab_size=512, max_position=512, **CONFIGS["gpt2"])
    model.reset_parameters(seed=1)
    ids = torch.randint(0, 512, (2, 64), device="cuda")
    model(ids, ids).backward()
    want = {n: p.grad.clone() for n, p in model.named_parameters()}
    model.zero_grad(set_to_none=True)
    loss = model(ids, ids)
    old = {}
    for n, p in model.named_parameters():
        old[n], p.data = p.data, p.data.clone()
    for t in old.values():
        t.fill_(float("nan"))                              # still allocated: whoever reads it finds no numbers
    loss.backward()
    for n, p in model.named_parameters():
        if n.startswith("blocks."):
            assert (p.grad.float() - want[n].float()).norm() <= 1e-2 * want[n].float().norm() + 1e-7, n
