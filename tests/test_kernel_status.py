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
