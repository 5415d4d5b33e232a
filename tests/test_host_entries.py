"""What the C entry points accept and refuse, on the host alone: every check here is made before a launch, so the
pointers are addresses that nothing reads."""

from mlkit_b200 import _native

F16, BF16, F32 = _native.F16, _native.BF16, _native.F32
POINTER, UNSUPPORTED = 1 << 20, -2


def rotated(x_dtype, rows=1, width=4096):
    return _native.library().mkb_gemv_hadamard(
        POINTER, POINTER, POINTER, POINTER, POINTER, None, POINTER, rows, 64, width, 128, 4, 16, x_dtype, F16,
        width // 2, width // 128, 1, -8.0, 1, None)


def test_rotation_on_load_takes_fp16_rows_only():
    for x_dtype in (BF16, F32):
        assert rotated(x_dtype) == UNSUPPORTED
        assert b"fp16" in _native.library().mkb_last_error()
    assert rotated(F16, width=14336) == UNSUPPORTED     # and no width with an odd factor
