"""The larger scratch of the attention backward is given up where it does not fit, and only then."""
import pytest
import torch


def test_scratch_falls_back_once(monkeypatch):
    from zen_repro_b200.ops import attention as A

    real, refused = torch.empty, []

    def room(n, **kw):
        if n > 1000:
            refused.append(n)
            raise torch.OutOfMemoryError("no room")
        return real(n, **kw)

    monkeypatch.setattr(torch, "empty", room)
    got = [A.scratch(most, least, torch.device("cpu")) for most, least in ((2000, 500), (800, 500), (500, 500))]
    assert [(t.numel(), k) for t, k in got] == [(500, 0), (800, 1), (500, 0)] and refused == [2000]
    with pytest.raises(torch.OutOfMemoryError):
        A.scratch(2000, 1500, torch.device("cpu"))
