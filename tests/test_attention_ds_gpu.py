"""Backward that keeps dS between its kernels against the one that works the scores out twice: ragged sequences, head sizes that do not
fill an atom, grouped heads, and which shapes take which."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bytes(B, S, hq, hkv, hd):
    from zen_repro_b200.ops import attention as A
    return A._flash_ds_bytes(B, S, hq, hd)


def test_when_it_is_kept():
    assert _bytes(1, 128, 512, 512, 64) == 0                         # one tile a head: nothing to share
    assert _bytes(1, 256, 2, 2, 64) == 0                             # few tiles
    assert _bytes(2, 1000, 12, 12, 64) == 2 * 12 * 36 * 32768
    assert _bytes(1, 8192, 32, 8, 128) == 32 * 64 * 65 // 2 * 32768
    assert _bytes(1, 8192, 32, 32, 80) == 0                          # small heads: more than the L2 holds
    assert _bytes(1, 65536, 32, 8, 128) == 0                         # more than its limit


@pytest.mark.parametrize("B,S,hq,hkv,hd", [(2, 1000, 12, 12, 64), (3, 129, 40, 40, 64), (6, 333, 8, 4, 80), (1, 2048, 6, 2, 128), (2, 700, 16, 1, 40),
                                           (1, 1153, 8, 4, 120), (7, 256, 16, 16, 8)])
def test_both_backwards_agree_with_fp32(B, S, hq, hkv, hd, monkeypatch):
    from zen_repro_b200.ops import attention as A

    torch.manual_seed(S + hd)
    assert _bytes(B, S, hq, hkv, hd) > 0
    scale = hd ** -0.5
    qkv = torch.randn(B * S, (hq + 2 * hkv) * hd, device="cuda").bfloat16()
    dout = torch.randn(B * S, hq * hd, device="cuda").bfloat16()
    out, lse2 = A.attention_fwd_kernel(qkv, B, S, hq, hkv, hd, scale)
    kept = A.attention_bwd_kernel(dout, qkv, out, lse2, B, S, hq, hkv, hd, scale)
    monkeypatch.setattr(A, "_flash_ds_bytes", lambda *a: 0)
    twice = A.attention_bwd_kernel(dout, qkv, out, lse2, B, S, hq, hkv, hd, scale)
    assert A.attention_error() == 0
    x = qkv.float().requires_grad_(True)
    (want,) = torch.autograd.grad(A.reference_attention(x, B, S, hq, hkv, hd, scale), x, dout.float())
    norm = want.norm()
    a, b = (kept.float() - want).norm() / norm, (twice.float() - want).norm() / norm
    # P and dS rounded to bf16 once each (2^-9 relative, at random), and the result
    assert a < 1e-2 and a < 1.02 * b + 1e-5, (a, b)
    q = hq * hd
    v = q + hkv * hd
    assert torch.equal(kept[:, v:], twice[:, v:])                    # dV is the same kernel's; dQ and dK hang on D, summed in another order
    for sl in (slice(0, q), slice(q, v)):
        assert (kept[:, sl].float() - twice[:, sl].float()).norm() <= 2e-3 * want[:, sl].norm()


# ------------------------------------------------------------------------------------------- where the scratch does not fit
class _Room:
    """torch.empty as on a device with room for ``left`` bytes a tensor."""

    def __init__(self, left):
        self.left, self.real, self.refused = left, torch.empty, 0

    def __call__(self, *size, **kw):
        t = self.real(*size, **dict(kw, device="meta"))
        if t.numel() * t.element_size() > self.left:
            self.refused += 1
            raise torch.OutOfMemoryError("no room")
        return self.real(*size, **kw)


def test_attention_runs_where_the_scratch_does_not_fit(monkeypatch):
    from zen_repro_b200.ops import attention as A

    B, S, hq, hkv, hd = 1, 1152, 16, 4, 128
    need = _bytes(B, S, hq, hkv, hd)
    assert need > 16 << 20
    qkv = torch.randn(B * S, (hq + 2 * hkv) * hd, device="cuda").bfloat16()
    dout = torch.randn(B * S, hq * hd, device="cuda").bfloat16()
    out, lse2 = A.attention_fwd_kernel(qkv, B, S, hq, hkv, hd, hd ** -0.5)
    room = _Room(need - 1)
    with monkeypatch.context() as m:
        m.setattr(torch, "empty", room)
        got = A.attention_bwd_kernel(dout, qkv, out, lse2, B, S, hq, hkv, hd, hd ** -0.5)
    assert room.refused == 1
    monkeypatch.setattr(A, "_flash_ds_bytes", lambda *a: 0)
    assert torch.equal(got, A.attention_bwd_kernel(dout, qkv, out, lse2, B, S, hq, hkv, hd, hd ** -0.5))
    assert A.attention_error() == 0


def test_block_runs_where_the_scratch_does_not_fit(monkeypatch):
    from zen_repro_b200.models import build_model
    from zen_repro_b200.ops import attention as A

    model = build_model("gpt2", device="cuda", num_layers=1)
    model.reset_parameters(seed=0)
    B, S = 4, 512
    cfg = model.cfg
    need = _bytes(B, S, cfg.num_heads, cfg.num_heads, cfg.head_dim)
    assert need > 0
    ids = torch.randint(0, cfg.vocab_size, (B, S), device="cuda")

    def grads():
        model.zero_grad()
        model(ids, ids).backward()
        return [p.grad.clone() for p in model.parameters() if p.grad is not None]

    kept = grads()
    asked = []
    real = A.scratch
    monkeypatch.setattr(A, "scratch", lambda most, least, dev: (asked.append(most - least), real(least, least, dev))[1])
    twice = grads()
    assert asked and asked[0] >= need
    for a, b in zip(kept, twice):                                    # as the two backwards of the attention alone
        assert (a.double() - b.double()).norm() <= 1e-2 * b.double().norm() + 1e-12
