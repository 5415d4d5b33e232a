"""The device encoder against the tensor route of the same format on the CPU: codes, packed stream, scales and
offsets are equal, bit for bit, whatever kernel the layout takes."""

import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu


def format_of(kind, bits, group, asym):
    import mlkit_b200 as mk

    values, integer = helpers.grid_values(kind, bits)
    grid = mk.grid.int(bits) if integer else mk.grid.values(torch.from_numpy(values), bits=bits)
    return mk.scaled(grid, group=group, asym=asym)


def same(got, expected, bits):
    import mlkit_b200 as mk

    assert torch.equal(got.codes.cpu(), expected.codes)
    assert torch.equal(got.params["scales"].cpu(), expected.params["scales"])
    assert (got.params["zero"] is None) == (expected.params["zero"] is None)
    if got.params["zero"] is not None:
        assert torch.equal(got.params["zero"].cpu(), expected.params["zero"])
    assert torch.equal(got.packed_stream(bits).cpu(), mk.pack(expected.codes, bits))
    assert got.bits == expected.bits and got.metadata == expected.metadata


@pytest.mark.parametrize("asym", [False, True])
@pytest.mark.parametrize("kind,bits", [("int", b) for b in range(2, 9)] + [("nf4", 4), ("codebook3", 3)])
def test_every_grid_and_type(kind, bits, asym):
    generator = torch.Generator().manual_seed(bits)
    for dtype in (torch.float16, torch.bfloat16, torch.float32):
        # a single run; a short last group; one row; rows that end inside a block
        for rows, width, group in ((1, 8, 8), (3, 264, 128), (1, 4096, 256), (67, 640, 64), (130, 896, 32), (5, 72, 16)):
            weight = (torch.randn(rows, width, generator=generator) * 0.02).to(dtype)
            weight[0, : width // 2] = 0
            weight[-1, -1] = 31.0
            weight[-1, 0] = -1e-6
            fmt = format_of(kind, bits, group, asym)
            same(fmt(weight.cuda()), fmt(weight), bits)


@pytest.mark.parametrize("bits", [2, 4, 8])
def test_quotients_at_rounding_boundaries(bits):
    """Weights at, just above and just below every half-integer multiple of their scale."""
    low, high = -(2 ** (bits - 1)), 2 ** (bits - 1) - 1
    half = torch.arange(low, high).float() + 0.5
    half = half.repeat(-(-62 // half.numel()))[:62] if bits < 7 else half
    rows = []
    for scale in (2.0**-24, 0.00099945068359375, 0.0123443603515625, 1.0, 3.001953125, 1000.0):
        exact = half * scale
        for nudged in (exact, torch.nextafter(exact, exact * 2), torch.nextafter(exact, exact * 0)):
            rows.append(torch.cat((torch.tensor([low * scale]), nudged, torch.zeros(256 - 1 - nudged.numel()))))
    weight = torch.stack(rows)
    fmt = format_of("int", bits, 256, False)
    same(fmt(weight.cuda()), fmt(weight), bits)


@pytest.mark.parametrize("kind,bits", [("int", 4), ("int", 8), ("nf4", 4), ("codebook3", 3)])
def test_narrow_groups_far_from_zero(kind, bits):
    """Their offset ends at fp16's largest value, the scale at its smallest, and w - offset over it overflows."""
    weight = torch.full((6, 128), 0.5)
    weight[0], weight[1], weight[2], weight[3], weight[4, 5] = 1e33, -1e33, 3e38, 2e31, 1e30
    weight[1, 7] = -1.0009765625e33
    weight[5, :64] = torch.linspace(-1.5e38, 1.5e38, 64)
    for dtype in (torch.float32, torch.bfloat16):
        for group in (64, 128):
            fmt = format_of(kind, bits, group, True)
            same(fmt(weight.to(dtype).cuda()), fmt(weight.to(dtype)), bits)


def test_layouts_and_refusals():
    import mlkit_b200 as mk

    generator = torch.Generator().manual_seed(1)
    base = (torch.randn(40, 520, generator=generator) * 0.02).half().cuda()
    views = (base[:, 8:264], base[:, 1:257].contiguous(), base.t()[:256].t(), base.flatten()[1:1 + 256 * 8].view(8, 256))
    for weight in views:
        for asym in (False, True):
            fmt = format_of("int", 4, 64, asym)
            same(fmt(weight), fmt(weight.cpu()), 4)
    for group, width in ((96, 192), (512, 1024), (None, 320), (128, 100)):   # the group kernel and the tensor route
        weight = (torch.randn(9, width, generator=generator) * 0.02).half()
        for asym in (False, True):
            fmt = mk.int(4, group=group, asym=asym)
            same(fmt(weight.cuda()), fmt(weight), 4)
    for value in (float("nan"), float("inf"), float("-inf")):
        weight = torch.zeros(4, 256, device="cuda")
        weight[3, 255] = value
        for asym in (False, True):
            with pytest.raises(ValueError):
                mk.int(4, group=64, asym=asym)(weight)
    trainable = torch.randn(4, 128, device="cuda", requires_grad=True)
    assert mk.int(4, asym=True)(trainable).params["scales"].requires_grad   # the tensor route stays differentiable
