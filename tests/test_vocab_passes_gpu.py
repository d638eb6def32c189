"""Edges of the fused passes around the vocabulary and the token positions: soft-capped cross-entropy (both CTA sizes), label shift and
count, position gradients, column sums whose vectors do not divide the CTA, rotation split into head groups, gradients that the
optimizer clears."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab,cap", [(3, 1000, 30.0), (300, 50_257, 0.0), (17, 256_001, 30.0), (1, 7, 5.0)])
def test_cross_entropy(rows, vocab, cap):
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(vocab)
    ld = (vocab + 7) // 8 * 8
    x = (torch.randn(rows, ld, device="cuda") * 8).bfloat16()
    labels = torch.randint(0, vocab, (rows,), device="cuda")
    labels[0] = -100 if rows > 1 else 0
    ref = x[:, :vocab].float().requires_grad_(True)
    z = cap * torch.tanh(ref / cap) if cap else ref
    want = F.cross_entropy(z, labels, reduction="none", ignore_index=-100)
    (g,) = torch.autograd.grad(want.sum() * 0.25, ref)
    inv = torch.full((1,), 0.25, device="cuda")
    loss, dl = E.cross_entropy(x.clone()[:, :vocab], labels, grad_scale=1.0, grad_scale_dev=inv, softcap=cap)
    torch.testing.assert_close(loss, want.detach(), atol=2e-2, rtol=2e-3)
    torch.testing.assert_close(dl.float(), g, atol=2e-3, rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,vocab,cap", [(5, 1003, 30.0), (9, 256_001, 30.0), (64, 4096, 5.0)])
def test_soft_capped_cross_entropy_near_the_cap(rows, vocab, cap, dtype):
    """Against 64 bits, with logits well into the flat part of the cap, where the gradient's factor 1 - tanh^2 cancels."""
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(vocab)
    ld = (vocab + 7) // 8 * 8
    x = (torch.randn(rows, ld, device="cuda") * 2 * cap).to(dtype)
    labels = torch.randint(0, vocab, (rows,), device="cuda")
    ref = x[:, :vocab].double().requires_grad_(True)
    z = cap * torch.tanh(ref / cap)
    want = F.cross_entropy(z, labels, reduction="none")
    (g,) = torch.autograd.grad(want.sum(), ref)
    capped = E.softcap_logits(x[:, :vocab], cap)
    loss, dl = E.cross_entropy(x.clone()[:, :vocab], labels, grad_scale=1.0, softcap=cap)
    # fp32: a tanh within 2 units and the roundings of cap * t * log2(e) make some 8 units of the cap in an exponent
    unit = 2.0**-24
    assert (loss - want).abs().max() <= 16 * cap * unit + 8 * unit * want.abs().max()
    assert (loss - F.cross_entropy(capped.double(), labels, reduction="none")).abs().max() <= 16 * cap * unit + 8 * unit * want.abs().max()
    # p (1 - t^2), |p - 1| at the label: 1 - t^2 is off by 4 units of 1, p by the exponent's; then the rounding to the result's type
    p = torch.softmax(z.detach(), -1)
    p[torch.arange(rows), labels] -= 1.0
    bound = p.abs() * 8 * unit + g.abs() * 32 * cap * unit + 2.0**-149
    if dtype == torch.bfloat16:
        bound = bound * (1 + 2.0**-8) + g.abs() * 2.0**-8
    p_abs = 16 * cap * unit * torch.softmax(z.detach(), -1) * (1 - (z.detach() / cap) ** 2)     # p near 1 at the label
    assert ((dl.double() - g).abs() <= bound + p_abs + 1e-37).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("masked", ["lowest", "-inf"])
@pytest.mark.parametrize("rows,vocab", [(3, 1000), (2, 20_003), (2, 256_001)])
def test_cross_entropy_of_masked_logits(rows, vocab, masked, dtype):
    """Whole vectors, and all that one thread sees first, of the type's lowest value or of -inf."""
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(vocab)
    x = (torch.randn(rows, (vocab + 7) // 8 * 8, device="cuda") * 3).to(dtype)
    x[:, : vocab - 70] = torch.finfo(dtype).min if masked == "lowest" else float("-inf")
    x[0, 5] = 1.0
    labels = torch.full((rows,), vocab - 3, device="cuda")
    ref = x[:, :vocab].double().requires_grad_(True)
    want = F.cross_entropy(ref, labels, reduction="none")
    (g,) = torch.autograd.grad(want.sum(), ref)
    loss, dl = E.cross_entropy(x.clone()[:, :vocab], labels, grad_scale=1.0)
    torch.testing.assert_close(loss.double(), want.detach(), atol=1e-5, rtol=1e-6)
    torch.testing.assert_close(dl.double(), g, atol=2e-6, rtol=1e-5 if dtype == torch.float32 else 2.0**-8)


@pytest.mark.parametrize("scale", [1.0, 1000.0])
def test_cross_entropy_of_large_fp32_logits(scale):
    """The loss to the rounding of a logit, the gradient to that rounding times its value: nothing is lost to log2(e)."""
    from zen_repro_b200.ops import elementwise as E

    torch.manual_seed(1)
    x = torch.randn(64, 4096, device="cuda") + scale
    labels = torch.randint(0, 4096, (64,), device="cuda")
    ref = x.double().requires_grad_(True)
    want = F.cross_entropy(ref, labels, reduction="none")
    (g,) = torch.autograd.grad(want.sum(), ref)
    loss, dl = E.cross_entropy(x.clone(), labels, grad_scale=1.0)
    # the log-sum-exp (at most scale + 10) is rounded once; a gradient's exponent, 14 at most, in its difference, its product and
    # log2(e), and the exponential is off by 2 units
    lse = 2.0 ** (math.floor(math.log2(scale + 10.0)) - 24)
    assert (loss - want).abs().max() <= lse + 2.0**-20
    assert ((dl.double() - g).abs() <= (lse + 2.0**-24 * (2.5 * 14 + 8)) * torch.softmax(ref.detach(), -1) + 2.0**-24 * g.abs()).all()


@pytest.mark.parametrize("bsz,seq,shift", [(1, 1, 1), (3, 77, 1), (2, 1500, 0)])
def test_label_prep(bsz, seq, shift):
    from zen_repro_b200.ops import elementwise as E

    labels = torch.randint(0, 50, (bsz, seq))
    labels[0, 0] = -100
    want = E.label_prep(labels, shift)
    lab, inv = E.label_prep(labels.cuda(), shift)
    assert torch.equal(lab.cpu().view(-1), want[0].view(-1))
    torch.testing.assert_close(inv.cpu().view(-1), want[1].view(-1))


@pytest.mark.parametrize("bsz,seq,d", [(1, 1, 8), (3, 50, 264), (5, 129, 768)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_pos_grad(bsz, seq, d, accumulate):
    from zen_repro_b200.ops import elementwise as E

    dy = torch.randn(bsz * seq, d, device="cuda").bfloat16()
    out = torch.randn(seq, d, device="cuda").bfloat16()
    want = dy.float().view(bsz, seq, d).sum(0) + (out.float() if accumulate else 0.0)
    E.pos_grad_(out, dy, bsz, accumulate)
    torch.testing.assert_close(out.float(), want, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("rows,cols", [(1, 8), (37, 384), (1000, 1016), (64, 2056)])
def test_colsum(rows, cols):
    from zen_repro_b200.ops import elementwise as E

    a = torch.randn(rows, cols, device="cuda").bfloat16()
    torch.testing.assert_close(E.colsum(a).float(), a.float().sum(0), atol=5e-2, rtol=1e-2)


@pytest.mark.parametrize("tokens,heads,hd,seq", [(5, 1, 8, 5), (64, 40, 128, 64), (700, 33, 80, 350), (9000, 3, 256, 4500)])
def test_rope_and_inverse(tokens, heads, hd, seq):
    from zen_repro_b200.ops import elementwise as E

    x = torch.randn(tokens, heads, hd).bfloat16()
    want = E.rope_(x.float().clone(), seq)
    got = E.rope_(x.cuda().clone(), seq)
    torch.testing.assert_close(got.float().cpu(), want, atol=3e-2, rtol=2e-2)
    torch.testing.assert_close(E.rope_(got, seq, inverse=True).float().cpu(), x.float(), atol=5e-2, rtol=2e-2)


@pytest.mark.parametrize("n", [1, 7, 65_537])
def test_optimizer_clears_what_it_has_used(n):
    from zen_repro_b200.optim.adamw import FusedAdamW

    torch.manual_seed(n)
    init, grad = torch.randn(n, device="cuda").bfloat16(), torch.randn(n, device="cuda").bfloat16()
    ps = []
    for clear in (False, True):
        p = torch.nn.Parameter(init.clone())
        p.grad = grad.clone()
        FusedAdamW([p], lr=1e-2).step(clear_grads=clear)
        ps.append(p)
    assert torch.equal(ps[0], ps[1]) and torch.equal(ps[0].grad, grad) and not ps[1].grad.any()
