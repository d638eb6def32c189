"""Which CPython extension the package loads: never one that another interpreter, or another source, was built for."""
import ctypes

import numpy as np
import pytest
import torch


@pytest.mark.parametrize("stamp", ["3.11.0 (another interpreter)", None])
def test_extension_of_another_interpreter_is_rebuilt(stamp, tmp_path, monkeypatch):
    from zen_repro_b200 import _native, build

    if not build.lib_path().exists():
        pytest.skip("native library not built")
    (tmp_path / build.LIBNAME).symlink_to(build.lib_path())
    (tmp_path / build.CALLNAME).write_bytes(b"not an extension of this interpreter")
    if stamp is not None:
        (tmp_path / "fastcall.stamp").write_text(stamp)
    monkeypatch.setattr(build, "LIBDIR", tmp_path)
    monkeypatch.setattr(_native, "_LIB", None)
    assert _native.lib().zen_block_size() > 0
    first = (tmp_path / build.CALLNAME).stat().st_mtime_ns
    monkeypatch.setattr(_native, "_LIB", None)
    assert _native.lib().zen_block_size() > 0
    assert (tmp_path / build.CALLNAME).stat().st_mtime_ns == first         # and then kept


def test_arguments_of_a_native_call():
    """Numbers and ctypes objects; nothing whose address could be taken for its value."""
    from zen_repro_b200 import _native, build

    if not build.lib_path().exists():
        pytest.skip("native library not built")
    f = _native.lib().zen_colsum_parts
    want = f(1000)
    assert want > 1 and f(ctypes.c_int(1000)) == want and f(True) == f(1) == f(None) + 1
    for bad in (np.int64(1000), np.zeros(4), torch.tensor(1000), b"1000", bytearray(8), "1000", [1000]):
        with pytest.raises(TypeError):
            f(bad)
    n = ctypes.c_int64(-1)
    assert _native.lib().zen_launch_count(ctypes.byref(n)) == 0 and n.value >= 0
    many = (ctypes.c_int64 * 2)(-1, -1)
    assert _native.lib().zen_launch_count(many) == 0 and many[0] >= 0 and many[1] == -1
    with pytest.raises(TypeError):
        f(*range(40))
