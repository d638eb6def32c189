"""Which CPython extension the package loads: never one that another interpreter, or another source, was built for."""
import pytest


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
