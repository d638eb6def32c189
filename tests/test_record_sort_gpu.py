"""What the record sort leaves, looked at by itself after whole calls: records of a tile in bucket order, the table of their runs, and
nothing lost; in small calls it is launched early, behind a partition that still runs, in large ones plainly."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TILE = 4096


@pytest.mark.parametrize("numel,P,density", [(262_144, 4, 0.4), (524_288, 2, 0.3), (140_001, 7, 0.7), (6_000_000, 4, 0.1), (30_000_000, 2, 0.05)])
def test_runs(numel, P, density):
    from zen_repro_b200.sparse.engine import VirtualSparseAllReduce

    eng = VirtualSparseAllReduce(numel, P, max_density=min(1.0, density * 1.2), methods=(3,))
    plan = eng.plan
    assert plan.cap_rec * P > 65_536 and plan.nslots > 1 << 14         # sorted, more than one bucket
    lg = 14 if plan.nslots <= 1 << 24 else 15
    tiles, buckets = -(-plan.cap_rec // TILE), -(-plan.nslots // (1 << lg))
    g = torch.Generator("cuda").manual_seed(numel)
    for _ in range(3):
        xs = [torch.where(torch.rand(numel, device="cuda", generator=g) < density, torch.randn(numel, device="cuda", generator=g), 0.0) for _ in range(P)]
        eng(xs, method=3)
        assert eng.status() == [0] * P
        values = [[] for _ in range(P)]
        for r, rank in enumerate(eng.ranks):
            counts = rank.metrics(eng.epoch)["recv_records"]
            seg = rank.seg[: buckets * P * tiles].view(buckets, P, tiles).long()
            for s, n in enumerate(counts):
                at = plan.off_rec + ((eng.epoch & 1) * P + s) * plan.cap_rec * 8
                rec = rank.region.view(r, at, n * 8, torch.int32).view(-1, 2)
                values[s].append(rec[:, 1])
                slots = rec[:, 0].long()
                assert (slots >= 0).all() and (slots < plan.nslots).all() and slots.unique().numel() == n
                where = torch.arange(n, device="cuda") // TILE * buckets + (slots >> lg)
                assert (where[1:] >= where[:-1]).all()
                used = -(-n // TILE)
                length = torch.bincount(where, minlength=used * buckets).view(used, buckets).t()
                assert torch.equal(seg[:, s, :used] >> 16, length)
                assert torch.equal(seg[:, s, :used] & 0xffff, torch.cumsum(length, 0) - length)
        for s, x in enumerate(xs):                                     # every non-zero of a source is with one of the owners
            assert torch.equal(torch.cat(values[s]).sort().values, x[x != 0].view(torch.int32).sort().values)
