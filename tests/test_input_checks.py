"""Ids and labels that the kernels would read out of bounds: converted where that is what is meant, else refused on the host."""
import pytest
import torch

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("name", ["tiny-gpt2", "tiny-llama"])
def test_32_bit_ids_and_labels(name, device):
    from zen_repro_b200.models import build_model

    model = build_model(name, device=device, dtype=torch.float32)
    model.reset_parameters(seed=1)
    ids = torch.randint(0, 1000, (3, 17), device=device)
    want, got = model(ids, ids), model(ids.int(), ids.int())
    assert torch.equal(want, got)
    got.backward()
    assert model.wte.grad.abs().sum() > 0


@pytest.mark.parametrize("device", DEVICES)
def test_sequence_beyond_the_position_table(device):
    from zen_repro_b200.models import build_model

    for name in ("tiny-gpt2", "tiny-opt"):
        model = build_model(name, device=device, dtype=torch.float32)
        assert model(torch.zeros(1, 64, dtype=torch.long, device=device)).shape == (1, 64, 1000)
        with pytest.raises(ValueError, match="position table"):
            model(torch.zeros(1, 65, dtype=torch.long, device=device))


@pytest.mark.gpu
def test_labels_on_the_host():
    from zen_repro_b200.ops import elementwise as E

    x = torch.randn(4, 16, device="cuda")
    with pytest.raises(ValueError, match="ids or labels"):
        E.cross_entropy(x, torch.zeros(4, dtype=torch.long))
    with pytest.raises(ValueError, match="5 labels for 4 rows"):
        E.cross_entropy(x, torch.zeros(5, dtype=torch.long, device="cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("first", [1, 8])
def test_logits_that_do_not_start_on_a_vector(dtype, first):
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(first)
    x = torch.randn(5, 4104, device="cuda").to(dtype)
    labels = torch.randint(0, 4000, (5,), device="cuda")
    whole, part = x[:, first:first + 4000].contiguous(), x.clone()[:, first:first + 4000]
    want, dw = E.cross_entropy(whole, labels, grad_scale=1.0)
    loss, dl = E.cross_entropy(part, labels, grad_scale=1.0)
    torch.testing.assert_close(loss, want, atol=1e-5, rtol=1e-6)
    torch.testing.assert_close(dl, dw, atol=1e-6, rtol=1e-5 if dtype == torch.float32 else 2.0**-7)
