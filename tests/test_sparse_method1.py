"""Method 1 takes its buckets only where the plan's scratch holds the runs of its records (plans that were not made for it) and where
the output takes 16-byte stores."""
import ctypes

import pytest
import torch

PLANS = [(500_000, 8, 0.12, (3,)), (524_288, 4, 0.12, (3,)), (400_000, 2, 0.25, (3,)), (524_288, 2, 0.12, (2, 3)), (500_000, 8, 0.06, (1, 3)),
         (524_288, 8, 1.0, (1,)), (16_384, 8, 0.12, (3,)), (16_383, 3, 0.12, (1,)), (524_289, 2, 0.12, (1,)), (20_000, 2, 0.02, (3,))]


def _words(plan, with_method1):
    from zen_repro_b200 import _native

    out = (ctypes.c_int64 * 2)()
    _native.lib().zen_sparse_scratch(plan.nslots, plan.cap_rec, plan.nranks, plan.numel if with_method1 else 0, ctypes.addressof(out))
    return int(out[0])


@pytest.mark.parametrize("numel,P,density,methods", PLANS)
def test_buckets_only_where_the_scratch_holds_them(numel, P, density, methods):
    from zen_repro_b200 import _native, build
    from zen_repro_b200.sparse.engine import SparsePlan, _Ctx

    if not build.lib_path().exists():
        pytest.skip("native library not built")
    plan = SparsePlan(numel, P, max_density=density, method1=1 in methods, forced_coo=2 in methods)
    c = _Ctx()
    c.nranks, c.cap_rec, c.numel, c.nslots = P, plan.cap_rec, numel, plan.nslots
    # what the kernels use: a run per tile of 4096 records of a source and bucket of 16 384 elements, above 65 536 record slots
    tiles, buckets = -(-plan.cap_rec // 4096), -(-numel // 16_384)
    used = tiles * P * buckets if buckets > 1 and plan.cap_rec * P > 65_536 else 0
    for words in (_words(plan, 1 in methods), used, max(used - 1, 0), 0):
        c.seg_words = words
        for addr in (0x7f0000000000, 0x7f0000000002, 0x7f0000000004, 0x7f0000000008):
            assert _native.lib().zen_sparse_method1_buckets(ctypes.byref(c), addr) == (16_384 <= numel <= 524_288 and used <= words and addr % 16 == 0)
    if 1 in methods and 16_384 <= numel <= 524_288:
        assert _words(plan, True) >= used


@pytest.mark.gpu
@pytest.mark.parametrize("numel,P,density,methods", PLANS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sums_and_the_words_behind_the_scratch(numel, P, density, methods, dtype):
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    eng = VirtualSparseAllReduce(numel, P, max_density=density, methods=methods)
    guarded = []
    for r in eng.ranks:
        buf = torch.full((r.seg.numel() + 8192,), 0x5AFEC0DE, dtype=torch.int32, device="cuda")
        r.ctx.seg = buf.data_ptr()
        guarded.append(buf[r.seg.numel():])
    g = torch.Generator("cuda").manual_seed(numel + P)
    share = 0.5 * density / (1 if 1 in methods else P)         # a plan without method 1 has slots for an owner's share of the records
    for _ in range(3):
        xs = [(torch.randn(numel, device="cuda", generator=g) * (torch.rand(numel, device="cuda", generator=g) < share)).to(dtype) for _ in range(P)]
        want = torch.zeros(numel, device="cuda", dtype=dtype)
        for x in xs:
            want = (want.float() + x.float()).to(dtype)
        outs = eng(xs, method=1)
        assert eng.status() == [0] * P
        assert all(torch.equal(o, want) for o in outs)
        assert all(bool((w == 0x5AFEC0DE).all()) for w in guarded)


@pytest.mark.gpu
@pytest.mark.parametrize("numel,P", [(20_000, 2), (524_288, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_stage_by_stage_into_any_element(numel, P, dtype, shift):
    """The stages launched one by one write to outputs that start at any element; what lies around them stays."""
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    eng = VirtualSparseAllReduce(numel, P, max_density=0.1, methods=(1,))
    g = torch.Generator("cuda").manual_seed(shift)
    xs = [(torch.randn(numel, device="cuda", generator=g) * (torch.rand(numel, device="cuda", generator=g) < 0.05)).to(dtype) for _ in range(P)]
    want = torch.zeros(numel, device="cuda", dtype=dtype)
    for x in xs:
        want = (want.float() + x.float()).to(dtype)
    eng.epoch += 1
    for r, x in zip(eng.ranks, xs):
        r.partition_push(x, eng.epoch, broadcast=True)
    for r in eng.ranks:
        buf = torch.full((numel + 16,), 7.0, device="cuda", dtype=dtype)
        r.scatter_sources(buf[shift:shift + numel], eng.epoch)
        assert torch.equal(buf[shift:shift + numel], want)
        assert bool((buf[:shift] == 7).all()) and bool((buf[shift + numel:] == 7).all())
    assert eng.status() == [0] * P
