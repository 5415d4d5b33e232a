"""What the C entry points accept and refuse, on the host alone.  The pointers are addresses that nothing may read, so
these tests do not run where a device would: there the calls that are accepted would launch."""

from pathlib import Path

import pytest
import torch

from mlkit_b200 import _native, kernels

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="an accepted call would launch on made-up addresses")
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


def test_many_row_transform_covers_what_its_rule_admits():
    """The wrapper's rule and the entry point agree at every factor and power (a call that gets as far as the launch
    fails there: no device)."""
    x, signs = torch.empty(64, dtype=torch.float16), torch.empty(64, dtype=torch.int8)
    for power in (64, 128, 256, 512, 1024, 2048):
        for factor in range(1, 50):
            for dtype, tag in ((torch.float16, F16), (torch.bfloat16, BF16), (torch.float32, F32)):
                status = _native.library().mkb_hadamard_mix(POINTER, POINTER, POINTER, POINTER, 64, factor * power, factor,
                                                            power, tag, 0, 1, None)
                admitted = kernels.mix_supported(x.to(dtype), signs, x, 64, factor, power)
                assert (status != UNSUPPORTED) == admitted, (factor, power, dtype)


def test_lanes_whose_wait_expired_keep_their_warp_barriers():
    """By reading the source, an expired wait being nothing to bring about on a device.  The decoders' loop has one warp
    barrier per block, behind both waits, and a lane that left at a wait meets the others at the barriers it leaves out;
    every other wait that ends a loop is voted on by the warp."""
    source = (Path(kernels.__file__).parent / "csrc" / "gemm_tile.cu").read_text()
    step = "i < count; i += kDecodeGroups)"
    decoders = source[source.index(step):source.index("// ================================ epilogue")]
    loop, left = decoders.split("for (; " + step)
    assert loop.count("__syncwarp();") == 1 and left.lstrip().startswith("__syncwarp();")
    assert loop.count("tile_wait(") == 2 and loop.rindex("tile_wait(") < loop.index("__syncwarp();") and loop.count("break;") == 2
    for line in source[source.index("// ================================ epilogue"):].splitlines():
        assert "tile_wait(" not in line or "__all_sync(0xffffffffu, tile_wait(" in line or "break" not in line


def test_tile_gemm_covers_what_its_rule_admits():
    for bits in range(1, 9):
        for group in (16, 32, 64, 96, 128, 256):
            for width in (64, 128, 192, 256, 896, 1000, 4096):
                status = _native.library().mkb_gemm_tile(
                    POINTER, POINTER, POINTER, POINTER, None, None, POINTER, 33, 64, width, group, bits, 1 << bits, F16, F16,
                    width * bits // 8, -(-width // group), 1, -float(1 << bits - 1), POINTER, 1 << 40, POINTER, None)
                admitted = kernels.tile_gemm_rows(64, width, group, bits, True) > 0
                assert (status != UNSUPPORTED) == admitted, (bits, group, width)


def test_tile_gemm_takes_more_rows_of_larger_weights():
    for bits in range(2, 7):
        for integer in (True, False):
            for width in (896, 1024, 4096, 14336):
                most = [kernels.tile_gemm_rows(outputs, width, 128, bits, integer) for outputs in (64, 512, 2048, 8192, 28672)]
                assert most == sorted(most) and 32 < most[0] <= most[-1] <= 1024
    # eight bits decode slowest: two tiles of rows cost more than writing the weight once
    assert kernels.tile_gemm_rows(4096, 4096, 128, 8, True) < kernels.tile_gemm_rows(4096, 4096, 128, 4, True)
