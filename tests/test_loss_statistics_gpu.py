"""Cross-entropy whose row statistics come out of the product that makes the logits: ragged rows and vocabularies, soft-capping, labels
that count for nothing, and what a gradient taken from the stored logits gives, against 64 bits."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

SHAPES = [(256, 256, 64), (300, 1001, 128), (777, 8, 72), (130, 4097, 200), (1000, 50257, 64), (257, 896, 64)]


@pytest.mark.parametrize("keep", [True, False])
@pytest.mark.parametrize("cap", [0.0, 5.0])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_against_64_bits(M, N, K, cap, keep):
    from zen_repro_b200.ops import elementwise as E
    from zen_repro_b200.ops import gemm as G

    torch.manual_seed(N + M)
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = (torch.randn(N, K, device="cuda") * 4 * K ** -0.5).bfloat16()
    labels = torch.randint(0, N, (M,), device="cuda")
    labels[::7] = -100
    labels[1] = N - 1
    vpad = (N + 7) // 8 * 8
    buf = torch.full((M, vpad), 9.0, device="cuda").bfloat16()
    out = buf[:, :N]
    part, target = G.gemm_nt_loss(a, b, labels, out=out if keep else None, softcap=cap)
    loss = torch.empty(M, device="cuda")
    lse = E.xent_finish(part, target, labels, N, loss, softcap=cap)
    assert G.gemm_error() == 0
    plain = torch.empty(M, vpad, device="cuda").bfloat16()[:, :N]
    G.gemm_nt(a, b, out=plain, pad_ok=True, bn=512)
    if keep:
        assert torch.equal(out, plain)
    else:
        assert (buf == 9.0).all()
    x = plain.double().requires_grad_(True)
    z = cap * torch.tanh(x / cap) if cap else x
    want = F.cross_entropy(z, labels, reduction="none")
    (g,) = torch.autograd.grad(want.sum(), x)
    # a loss is a difference of two numbers of the logits' size, each within a few units of 2^-24 of that; sums of N exponentials
    # of relative error 2^-22 in fp32 add as little
    unit = 2.0 ** -24
    bound = 16 * unit * (z.detach().abs().max() + 16)
    assert (loss - want).abs().max() <= bound
    assert (lse - torch.logsumexp(z.detach(), -1)).abs().max() <= bound
    if keep:
        inv = torch.full((1,), 0.25, device="cuda")
        E.xent_grad_(out, labels, lse, inv, softcap=cap)
        err = (out.double() - g * 0.25).abs()
        p = torch.softmax(z.detach(), -1)
        assert (err <= g.abs() * 0.25 * 2.0 ** -8 + (p + 1e-3 * g.abs()) * 64 * unit * (z.detach().abs().max() + 16) + 1e-37).all()


def test_a_loss_that_is_not_finite_stays_so():
    """A NaN or an infinity in the activations reaches the loss of its row and of no other."""
    from zen_repro_b200.ops import elementwise as E
    from zen_repro_b200.ops import gemm as G

    torch.manual_seed(3)
    M, N, K = 256, 1000, 64
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    a[5, 0], a[9, 0] = float("nan"), float("inf")
    labels = torch.randint(0, N, (M,), device="cuda")
    loss = torch.empty(M, device="cuda")
    part, target = G.gemm_nt_loss(a, b, labels)
    E.xent_finish(part, target, labels, N, loss)
    bad = ~torch.isfinite(loss)
    assert bad[5] and bad[9] and int(bad.sum()) == 2


@pytest.mark.parametrize("softcap", [0.0, 30.0])
@pytest.mark.parametrize("rows", [64, 300, 1000, 1023, 1024, 1100, 2047, 2048])
def test_loss_function_equals_the_separate_passes(rows, softcap, monkeypatch):
    from zen_repro_b200.ops import gemm as G
    from zen_repro_b200.ops.autograd import lm_head_loss

    torch.manual_seed(rows)
    V, d = 5003, 256
    h = torch.randn(rows, d, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(V, d, device="cuda") * 0.1).bfloat16().requires_grad_(True)
    labels = torch.randint(0, V, (rows,), device="cuda")
    labels[::5] = -100

    def run():
        loss = lm_head_loss(h, w, labels, chunk_tokens=1024, unit_grad=False, softcap=softcap)
        gh, gw = torch.autograd.grad(loss, (h, w))
        training.append(len(ran))
        with torch.no_grad():
            quiet = lm_head_loss(h, w, labels, chunk_tokens=1024, softcap=softcap)
        return loss.detach(), quiet, gh, gw

    ran, training = [], []
    real = G.gemm_nt_loss
    monkeypatch.setattr(G, "gemm_nt_loss", lambda *a, **k: ran.append(1) or real(*a, **k))
    one = run()
    # in training the chunks of 1024 rows, and those alone; without a gradient every chunk whose product is of that kind
    sizes = [min(1024, rows - s) for s in range(0, rows, 1024)]
    kind = [G.makes_loss_statistics(h.detach()[:n], w.detach()) for n in sizes]
    assert rows < 1024 or kind[0]
    assert training == [sum(n == 1024 for n in sizes)] and len(ran) == training[0] + sum(kind)
    monkeypatch.setattr(G, "makes_loss_statistics", lambda a, b: False)
    two = run()
    assert abs(one[0] - two[0]) <= 1e-5 * two[0] and abs(one[1] - one[0]) <= 1e-6 * one[0]
    for x, y in zip(one[2:], two[2:]):
        assert (x.double() - y.double()).norm() <= 4e-3 * y.double().norm()       # bf16 gradients of the same fp32 softmax


@pytest.mark.parametrize("labels", [lambda: torch.zeros(299, dtype=torch.int64, device="cuda"), lambda: torch.zeros(600, dtype=torch.int64, device="cuda"),
                                    lambda: torch.zeros(300, dtype=torch.int32, device="cuda"), lambda: torch.zeros(300, dtype=torch.int64),
                                    lambda: torch.zeros(600, dtype=torch.int64, device="cuda")[::2]])
def test_labels_that_the_kernel_would_misread_are_refused(labels):
    from zen_repro_b200 import _native
    from zen_repro_b200.ops import gemm as G

    a, b = torch.randn(300, 64, device="cuda").bfloat16(), torch.randn(1000, 64, device="cuda").bfloat16()
    before = _native.launch_count()
    with pytest.raises(ValueError):
        G.gemm_nt_loss(a, b, labels())
    assert _native.launch_count() == before


@pytest.mark.parametrize("dead", [64, 128, 700, 1000])
def test_infinite_logits_are_capped_too(dead):
    """Soft-capped logits of -inf are -cap: boxes, pieces and whole rows of nothing else still count."""
    from zen_repro_b200.ops import elementwise as E
    from zen_repro_b200.ops import gemm as G

    torch.manual_seed(dead)
    M, N, K, cap = 256, 1000, 64, 5.0
    a = (torch.rand(M, K, device="cuda") + 0.1).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.1 - 0.6).bfloat16()           # the others lie near -cap as well
    b[:dead] = float("-inf")
    labels = torch.randint(0, N, (M,), device="cuda")
    loss = torch.empty(M, device="cuda")
    part, target = G.gemm_nt_loss(a, b, labels, softcap=cap)
    lse = E.xent_finish(part, target, labels, N, loss, softcap=cap)
    z = cap * torch.tanh(G.gemm_nt(a, b, bn=512).double() / cap)
    assert (z[:, :dead] == -cap).all()
    bound = 16 * 2.0 ** -24 * (cap + 16)                                    # as in test_against_64_bits
    assert (lse - torch.logsumexp(z, -1)).abs().max() <= bound
    assert (loss - F.cross_entropy(z, labels, reduction="none")).abs().max() <= bound
