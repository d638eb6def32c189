"""The norm kernels read and write 16 bytes at a time, so an operand that starts anywhere else is refused before anything is launched."""
import pytest

BASE = 0x7f0000000000                       # never dereferenced: the calls below end on the host


@pytest.fixture
def lib():
    from zen_repro_b200 import _native, build

    if not build.lib_path().exists():
        pytest.skip("native library not built")
    before = _native.launch_count()
    yield _native.lib()
    assert _native.launch_count() == before


@pytest.mark.parametrize("dtype", [0, 1, 2])
@pytest.mark.parametrize("cols", [768, 3072, 4096, 8192])
@pytest.mark.parametrize("off", [2, 4, 8])
def test_operands_off_16_bytes_are_refused(lib, dtype, cols, off):
    rows, stat = 64, BASE + (1 << 32)
    for bad in range(6):                    # x, residual, weight, bias, y, h
        x, res, w, b, y, h = (BASE + i * (1 << 24) + (off if i == bad else 0) for i in range(6))
        assert lib.zen_norm_fwd(x, res, w, b, y, h, stat, stat, rows, cols, 1e-5, 1, 0, dtype, 0) == -3
    for bad in range(5):                    # dy, h, weight, residual gradient, dh
        dy, h, w, dres, dh = (BASE + i * (1 << 24) + (off if i == bad else 0) for i in range(5))
        assert lib.zen_norm_bwd_sums(dy, h, w, stat, stat, dres, dh, stat, stat, 0, 0, 0, rows, cols, 1, 0, 0, dtype, 1, 0) == -3
