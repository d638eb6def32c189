"""Where the plan of a forward pass without a backward cuts K, and where it never does."""
import pytest

from zen_repro_b200.ops import gemm as G

SHAPES = [(2304, 768), (768, 768), (3072, 768), (768, 3072), (5120, 3072), (3072, 3072), (16384, 3072), (3072, 8192), (2560, 10240),
          (9216, 2304), (2304, 9216), (8, 8), (264, 4096)]


@pytest.mark.parametrize("N,K", SHAPES)
def test_forward_only_plan(N, K):
    for M in [1, 2, 37, 64, 127, 128, 129, 130, 255, 256, 257, 300, 333, 511, 512, 513, 600, 777, 1024, 1500, 4096, 8192, 32768]:
        kind, how, *whole = G.plan_forward_only(M, N, K)
        assert kind in ("one", "pair")                                  # clusters never share K here
        slices = how if kind == "pair" else 1
        assert slices == G.split_k_choice(M, N, K) and slices <= 2
        if M < 256:
            assert slices == 1
        halves_allowed = kind == "pair" and slices == 1 and not whole    # the launcher may cut the tiles of a partly filled last round
        tiles = -(-M // 256) * -(-N // 256)
        fill = M * N / (65536.0 * -(-tiles // G._clusters()) * G._clusters())
        if halves_allowed:
            assert M >= 512 and N >= 256 and fill >= 0.6


def test_the_order_of_summation_depends_on_the_token_count():
    """Stated where the plan is made: 3072 columns of depth 8192 take two slices at 256, 400 and 512 tokens, none at 300, 777, 1024."""
    cut = [G.plan_forward_only(M, 3072, 8192)[1] == 2 and G.plan_forward_only(M, 3072, 8192)[0] == "pair" for M in (256, 400, 512, 300, 777, 1024)]
    assert cut == [True, True, True, False, False, False]
