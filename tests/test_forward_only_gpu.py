"""Passes without gradients (validation, scoring): logits and losses of every family against the same model in fp32, and against
what a recorded forward gives.  Full widths, two layers, from one token to the first counts that cut K."""
import copy

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

VOCAB = 1000
FAMILIES = ["gpt2", "facebook/opt-2.7b", "meta-llama/Llama-3.2-3B", "gemma-2b", "google/gemma-2-2b"]


@pytest.fixture(scope="module", params=FAMILIES)
def models(request):
    from zen_repro_b200.models import build_model

    kw = dict(num_layers=2, vocab_size=VOCAB, max_position=1024)
    model = build_model(request.param, device="cuda", **kw)
    model.reset_parameters(seed=1)
    with torch.no_grad():
        for n, p in model.named_parameters():
            if n.endswith("_b"):
                p.normal_(0.0, 0.02)
    exact = build_model(request.param, device="cuda", dtype=torch.float32, **kw)
    exact.load_state_dict(copy.deepcopy(model.state_dict()))
    yield model, exact
    del model, exact
    torch.cuda.empty_cache()


def _error(got, want):
    return float((got.double() - want.double()).norm() / want.double().norm())


@pytest.mark.parametrize("bsz,seq", [(1, 1), (1, 37), (2, 64), (1, 256), (1, 300), (3, 333), (2, 512)])
def test_logits_and_loss(models, bsz, seq, monkeypatch):
    """bf16 keeps 8 bits: a result of about ten roundings a layer, each 2^-9 / sqrt(3) of its value, is off by half a percent
    after two layers; 2 % leaves room for what cancels.  No worse than the recorded forward by more than the draw of the roundings."""
    from zen_repro_b200.ops import block, gemm

    model, exact = models
    ids = torch.randint(0, VOCAB, (bsz, seq), device="cuda", generator=torch.Generator("cuda").manual_seed(seq))
    calls = []
    real = block.run
    monkeypatch.setattr(block, "run", lambda *a: calls.append(1) or real(*a))
    with torch.no_grad():
        want, logits = exact(ids), model(ids)
        assert len(calls) == 2
        loss, want_loss = model(ids, ids), exact(ids, ids)
    recorded = model(ids)
    assert recorded.requires_grad and not logits.requires_grad
    assert logits.shape == (bsz, seq, VOCAB) and logits.dtype == recorded.dtype
    assert gemm.gemm_error() == 0
    here, there = _error(logits, want), _error(recorded.detach(), want)
    assert here < 0.02 and here < 1.5 * there + 1e-3, (here, there)
    if seq > 1:
        # the mean of independent errors of the logits' size, and never less than one rounding of the loss
        by_hand = F.cross_entropy(logits[:, :-1].reshape(-1, VOCAB).double(), ids[:, 1:].reshape(-1))
        assert abs(float(loss - by_hand)) < 2e-3 and abs(float(loss - want_loss)) < 1e-2
        trained = model(ids, ids)
        assert trained.requires_grad and abs(float(loss - trained.detach())) < 5e-3


def test_softcap_logits():
    from zen_repro_b200.ops import elementwise as E

    for dtype in (torch.float32, torch.bfloat16):
        for rows, cols, ld in ((1, 1, 8), (3, 1003, 1008), (130, 4096, 4096)):
            x = (torch.randn(rows, ld, device="cuda") * 40).to(dtype)[:, :cols]
            got, want = E.softcap_logits(x, 30.0), 30.0 * torch.tanh(x.double() / 30.0)
            # a quotient, a tanh within 2 units and a product
            assert got.dtype == torch.float32 and ((got - want).abs() <= 4 * 2.0**-23 * want.abs() + 1e-37).all()
