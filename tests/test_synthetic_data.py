"""Token streams of large seeds: any seed a generator takes makes a stream, and one of its own."""
import pytest
import torch

from zen_repro_b200.data.synthetic import ZipfTokenStream


@pytest.mark.parametrize("seed", [2**31, 2**31 + 1, 2**32 - 1, 2**63, -(2**31)])
@pytest.mark.parametrize("dp_rank", [0, 7])
def test_any_seed_makes_a_stream(seed, dp_rank):
    first, again = (ZipfTokenStream(1000, 16, 2, seed=seed, dp_rank=dp_rank, pin=False) for _ in range(2))
    a, b = next(first)["input_ids"], next(again)["input_ids"]
    assert torch.equal(a, b)
    other = ZipfTokenStream(1000, 16, 2, seed=seed + 1, dp_rank=dp_rank, pin=False)
    assert not torch.equal(a, next(other)["input_ids"])
    assert not torch.equal(a, next(first)["input_ids"])


@pytest.mark.parametrize("seed,dp_rank", [(0, 0), (17, 3), (9_000_000, 7), (-5, 1)])
def test_small_seeds_keep_their_streams(seed, dp_rank):
    vocab, step = 1000, 4
    s = ZipfTokenStream(vocab, 16, 2, seed=seed, dp_rank=dp_rank, pin=False)
    s.load_state_dict({"step": step})
    g = torch.Generator().manual_seed((seed * 1_000_003 + dp_rank) * 1_000_003 + step)
    u = torch.rand(32, generator=g, dtype=torch.float64)
    assert torch.equal(next(s)["input_ids"].view(-1), torch.searchsorted(s.cdf, u).clamp_(max=vocab - 1))
