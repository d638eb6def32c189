"""The tiles of a partly filled last round as two halves of K: where the workspace holds what they exchange, and nothing beyond it is
written."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

HALVES = 2 * 2 * 128 * 256                  # floats that the two halves of a tile exchange; 16 counters beside them


def _clusters():
    return torch.cuda.get_device_properties(0).multi_processor_count // 2


def _group(pairs, ws_floats, n_counters):
    """a' b of each pair in one launch, with a workspace of that size between guard words."""
    from zen_repro_b200 import _native
    from zen_repro_b200.ops import gemm as G

    ws = torch.full((ws_floats + 4096,), 3.0, device="cuda")
    cnt = torch.zeros(n_counters + 64, dtype=torch.int32, device="cuda")
    outs = [torch.empty(a.shape[1], b.shape[1], dtype=torch.bfloat16, device="cuda") for a, b in pairs]
    descs = (G._GemmDesc * len(pairs))()
    for i, ((a, b), c) in enumerate(zip(pairs, outs)):
        descs[i] = G._GemmDesc(a.data_ptr(), b.data_ptr(), c.data_ptr(), a.shape[1], b.shape[1], a.shape[0], a.stride(0), b.stride(0), c.stride(0), 0, 0)
    rc = _native.lib().zen_gemm_bf16_2cta_group(descs, len(pairs), 1, 1, ws.data_ptr() if ws_floats else 0, ws_floats, cnt.data_ptr(), n_counters,
                                                _native.stream_ptr())
    assert rc == 0 and G.gemm_error() == 0
    assert bool((ws[ws_floats:] == 3.0).all()) and not bool(cnt.any())
    return outs


def _pair(k, m, n):
    return torch.randn(k, m, device="cuda").bfloat16(), torch.randn(k, n, device="cuda").bfloat16()


def _sum_of_halves(a, b):
    """a' b as the two halves of K, each summed in fp32 by a launch of its own, then added and rounded."""
    from zen_repro_b200.ops import gemm as G

    half = (a.shape[0] // 64 + 1) // 2 * 64
    parts = [G.gemm_tn(a[s], b[s], out_dtype=torch.float32, bn=512) for s in (slice(0, half), slice(half, None))]
    return (parts[0] + parts[1]).bfloat16()


@pytest.mark.parametrize("k", [1024, 2112])
@pytest.mark.parametrize("missing", [0, 1])
def test_a_workspace_for_the_tiles_at_hand_is_enough(k, missing):
    torch.manual_seed(k)
    rem = 5
    pairs = [_pair(k, (_clusters() + rem) * 256, 256)]
    (whole,) = _group(pairs, 0, 0)
    for floats, counters in ((rem * HALVES - missing, rem * 16), (rem * HALVES, rem * 16 - missing)):
        (got,) = _group(pairs, floats, counters)
        cut = (got != whole).any(1).view(-1, 256).any(1)            # per tile
        # fp32 sums in another order differ somewhere in every tile of 65 536 elements
        assert int(cut.sum()) == (0 if missing else rem)
        if not missing:
            assert torch.equal(got.view(-1, 256, 256)[cut], _sum_of_halves(*pairs[0]).view(-1, 256, 256)[cut])


@pytest.mark.parametrize("k", [1024, 2240, 2248, 4096])
@pytest.mark.parametrize("shapes", [[(512, 512), (512, 256)], [(256, 256)], [(768, 768), (768, 1024), (1000, 776)]])
def test_groups_of_less_than_a_round_are_cut(shapes, k):
    """Weight gradients of a narrow layer: no split-K plan sees a group, so the launch itself shares the idle clusters out."""
    torch.manual_seed(len(shapes))
    pairs = [_pair(k, m, n) for m, n in shapes]
    tiles = sum(-(-m // 256) * -(-n // 256) for m, n in shapes)
    assert 2 * tiles <= _clusters()
    whole = _group(pairs, 0, 0)
    for got, one, (a, b) in zip(_group(pairs, tiles * HALVES, tiles * 16), whole, pairs):
        assert torch.equal(got, _sum_of_halves(a, b) if k > 35 * 64 else one)


@pytest.mark.parametrize("n", [28672, 40960])
def test_the_caller_says_what_no_product_reads(n):
    """Rows beyond the last whole 256 in an output whose last round is cut along K: transposed tiles, and with them another order of
    summation, only where the caller allows it, whatever the width."""
    from zen_repro_b200 import _native
    from zen_repro_b200.ops import gemm as G

    torch.manual_seed(n)
    # 44 rows over; narrow tiles shorten the rounds of both widths
    a, b = torch.randn(300, 1024, device="cuda").bfloat16(), torch.randn(n, 1024, device="cuda").bfloat16()
    tiles, per = 2 * (n // 256), _clusters()
    assert tiles > per and 0 < 2 * (tiles % per) <= per
    inner, last = (G.gemm_nt(a, b, bn=512, last=flag) for flag in (False, True))
    old = _native.lib().zen_gemm2_tail_split(0)
    try:
        whole = G.gemm_nt(a, b, bn=512)
    finally:
        _native.lib().zen_gemm2_tail_split(old)
    changed = (inner != whole).view(300, n // 256, 256).any(2)
    assert 0 < int(changed.any(0).sum()) < n // 256                  # the tiles of the last round alone
    assert torch.equal(last, whole)


def test_logits_say_so(monkeypatch):
    from zen_repro_b200.models import build_model
    from zen_repro_b200.ops import gemm as G

    model = build_model("gpt2", device="cuda", num_layers=1)
    model.reset_parameters(seed=0)
    ids = torch.randint(0, model.cfg.vocab_size, (1, 300), device="cuda")
    seen = []
    real = G.gemm_nt
    monkeypatch.setattr(G, "gemm_nt", lambda a, b, *r, **k: (seen.append((b.shape[0], bool(k.get("last")))), real(a, b, *r, **k))[1])
    model(ids)
    model(ids, ids)
    assert {w for w, flag in seen if flag} == {model.cfg.vocab_size} == {w for w, _ in seen if w > 10_000}
