"""Owner's sums in shared memory: every bucket shape (records read by every CTA, sorted tiles, 32 768-slot buckets, too many slots for
buckets), formats, types and densities against the dense sum; in rank order bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(n, P, density, dtype, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    keep = lambda: torch.rand(n, device="cuda", generator=g) < density
    return [torch.where(keep(), torch.randn(n, device="cuda", generator=g), torch.zeros((), device="cuda")).to(dtype) for _ in range(P)]


def _shape(eng):
    import ctypes
    from zen_repro_b200 import _native
    out = (ctypes.c_int64 * 2)()
    _native.lib().zen_sparse_scratch(eng.plan.nslots, eng.plan.cap_rec, eng.plan.nranks, 0, ctypes.addressof(out))
    return ("sorted" if out[0] > 1 else "read") if not out[1] else "global"


@pytest.mark.parametrize("n,P,density,kind", [
    (16_384 * 2, 2, 0.05, "read"),                 # one whole bucket an owner
    (16_384 * 2 + 130, 2, 0.05, "read"),           # a second bucket of one block
    (400_000, 3, 0.02, "read"),
    (3_000_017, 8, 0.05, "sorted"),
    (1_000_003, 2, 0.4, "sorted"),                 # dense mode: more than one record per four slots
    (20_000_001, 1, 0.01, "sorted"),               # 32 768-slot buckets
    (34_000_000, 1, 0.003, "global"),
])
@pytest.mark.parametrize("method", [2, 3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_matches_the_dense_sum(n, P, density, kind, method, dtype):
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    eng = VirtualSparseAllReduce(n, P, max_density=min(1.0, 1.3 * density), methods=(method,), deterministic=True)
    assert _shape(eng) == kind
    for call in range(3):                          # both parities of the record slots
        xs = _inputs(n, P, density * (1.0, 0.1, 0.9)[call], dtype, 10 * call + P)
        want = torch.zeros(n, device="cuda")
        for x in xs:
            want += x.float()
        outs = eng(xs, method=method)
        assert eng.status() == [0] * P
        for o in outs:
            assert torch.equal(o, want.to(dtype))


@pytest.mark.parametrize("n,P", [(50_000, 2), (3_000_017, 8)])
def test_full_buckets_and_staged_calls(n, P):
    """Every slot taken, one block of 64 taken by all, nothing at all; and the stages launched one by one give the same."""
    from zen_repro_b200.sparse import engine as E

    eng = E.VirtualSparseAllReduce(n, P, max_density=1.0, methods=(3,), deterministic=True)
    one = torch.zeros(n, device="cuda")
    one[64:128] = 1.5
    for xs in ([torch.randn(n, device="cuda") for _ in range(P)], [one.clone() for _ in range(P)], [torch.zeros(n, device="cuda")] * P):
        want = torch.zeros(n, device="cuda")
        for x in xs:
            want += x
        outs = eng(xs, method=3)
        assert eng.status() == [0] * P
        assert all(torch.equal(o, want) for o in outs)
        eng.epoch += 1
        staged = [torch.empty(n, device="cuda") for _ in range(P)]
        for r, x in zip(eng.ranks, xs):
            r.partition_push(x, eng.epoch)
        for r in eng.ranks:
            r.owner_reduce(eng.epoch, torch.float32, True)
        for r in eng.ranks:
            r.gather_push(eng.epoch, torch.float32, E.FMT_BITMAP)
        for r, o in zip(eng.ranks, staged):
            r.densify(o, eng.epoch, E.FMT_BITMAP)
        assert eng.status() == [0] * P
        assert all(torch.equal(o, want) for o in staged)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("method", [2, 3, "auto"])
def test_any_order(dtype, method):
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    n, P = 2_000_001, 4
    eng = VirtualSparseAllReduce(n, P, max_density=0.2, methods=(2, 3))
    xs = _inputs(n, P, 0.1, dtype, 5)
    want = torch.zeros(n, device="cuda", dtype=torch.float64)
    for x in xs:
        want += x.double()
    outs = eng(xs, method=method)
    assert eng.status() == [0] * P
    # up to four fp32 adds, one rounding to the type
    unit = {torch.float32: 2.0 ** -24, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    bound = sum(x.double().abs() for x in xs) * 3 * 2.0 ** -24 + want.abs() * unit + (2.0 ** -24 if dtype is torch.float16 else 0.0)
    for o in outs:
        assert ((o.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("n,P,density", [(1, 2, 1.0), (16_384, 3, 0.05), (16_385, 2, 0.5), (40_003, 8, 0.02), (524_288, 8, 0.05), (524_289, 2, 0.05)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_method_1_adds_source_after_source(n, P, density, dtype):
    """The sum is rounded to the type after every source, in rank order: bit for bit, whatever the bucket shape."""
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    eng = VirtualSparseAllReduce(n, P, max_density=min(1.0, 1.3 * density), methods=(1,))
    for call in range(3):
        xs = _inputs(n, P, density * (1.0, 0.1, 0.9)[call], dtype, 3 * call + P)
        want = torch.zeros(n, device="cuda", dtype=dtype)
        for x in xs:
            want = (want.float() + x.float()).to(dtype)
        outs = eng(xs, method=1)
        assert eng.status() == [0] * P
        for o in outs:
            assert torch.equal(o, want)
