"""Every error flag that a kernel of the library can set reaches ``Trainer.check_health``."""
import re
from types import SimpleNamespace

import pytest
import torch

from zen_repro_b200 import build

FLAGS = sorted({f for src in build.sources() for f in re.findall(r"^int (zen_\w+_error)\(\)", src.read_text(), re.M)})


def test_the_flags_are_found():
    assert {"zen_gemm2_error", "zen_flash_error", "zen_norm_error"} <= set(FLAGS)


@pytest.mark.parametrize("flag", FLAGS)
def test_flag_reaches_the_health_check(flag, monkeypatch):
    from zen_repro_b200 import _native
    from zen_repro_b200.trainer import Trainer

    fake = SimpleNamespace(**{f: (lambda f=f: 7 if f == flag else 0) for f in FLAGS})
    monkeypatch.setattr(_native, "lib", lambda: fake)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    module = SimpleNamespace()
    trainer = SimpleNamespace(device=torch.device("cuda"), model=SimpleNamespace(module=module, unwrap=lambda: module))
    got = Trainer.check_health(trainer, raise_on_error=False)
    assert [v for v in got.values() if v] == [7]
    with pytest.raises(RuntimeError, match="status words"):
        Trainer.check_health(trainer)


# ------------------------------------------------------------------------------ bounded waits for other ranks' mail
def _kernels():
    for name in ("sparse_kernels.cu", "sparse_row_kernels.cu"):
        for body in (build.CSRC / name).read_text().split("__global__")[1:]:
            if re.search(r"\w*_wait(_epoch)?\(", body.split("\n}\n")[0]):
                yield pytest.param(body.split("\n}\n")[0], id=re.search(r"(\w+)\(const", body).group(1))


def _guarded(body):
    """What a body does in its first CTA alone."""
    for m in re.finditer(r"if \([^\n]*blockIdx\.x == 0[^\n{]*\)\s*(\{)?", body):
        rest = body[m.end():]
        yield rest[:rest.index("}" if m.group(1) else ";")]


@pytest.mark.parametrize("body", list(_kernels()))
def test_every_cta_reports_its_own_wait(body):
    """CTAs of one kernel wait for a mail each for itself, so one may give up on what the first one saw; its records are then missing
    and the status has to say so."""
    assert re.search(r"ZEN_TIMEOUT|records_wait\(", body) and "atomicOr(c.status" in body
    assert not any("local_status" in g for g in _guarded(body))


@pytest.mark.gpu
@pytest.mark.parametrize("numel,P,stages", [(10_000, 2, "reduce"), (4_000_000, 4, "reduce gather"), (60_000, 2, "gather"), (300_000, 8, "scatter"), (900_000, 2, "scatter")])
def test_a_mail_that_never_comes_is_reported(numel, P, stages):
    from zen_repro_b200.sparse import engine as E

    eng = E.VirtualSparseAllReduce(numel, P, max_density=0.2, methods=(1,) if stages == "scatter" else (3,))
    x = torch.zeros(numel, device="cuda")
    x[::50] = 1.0
    eng.epoch += 1
    for r in eng.ranks[:-1]:
        r.partition_push(x, eng.epoch, broadcast=stages == "scatter")
    first = eng.ranks[0]
    for stage in stages.split():
        if stage == "reduce":
            first.owner_reduce(eng.epoch, x.dtype)
        elif stage == "gather":
            first.gather_push(eng.epoch, x.dtype)
        else:
            first.scatter_sources(torch.empty_like(x), eng.epoch)
        assert first.read_status() & E.ST_TIMEOUT, stage
