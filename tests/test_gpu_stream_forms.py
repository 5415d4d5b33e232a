"""The streaming matvec over every codec form AUTO gives it, for both activation types, against a 64-bit
reconstruct-then-matmul of the same codes; and the forms it must leave to the general kernel.

Tolerances.  A result is rounded once to the activation type (half a unit of the last place: at most 2^-8 of the
value for bf16's 8 significant bits, 2^-11 for fp16's 11).  With bf16 nothing else is rounded to 16 bits, so the
bound is 2^-8 plus fp32 accumulation.  With fp16 a
table level and its product with a scale are rounded too: three roundings of at most 2^-11.
"""

import numpy as np
import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu
BOUND = {torch.bfloat16: 2.0**-8 * 1.001, torch.float16: 3 * 2.0**-11}
FORMS = [("int", b, 128, False) for b in range(2, 9)] + [("int", 4, 64, False), ("int", 4, 32, False)] + \
        [("int", 4, g, True) for g in (128, 64, 32)] + [("nf4", 4, 64, False), ("nf4", 4, 128, False)] + \
        [("codebook3", 3, 64, False), ("codebook3", 3, 128, False)]


def layer_of(kind, bits, group, zeros, outputs, width, seed=0):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    values = torch.from_numpy(helpers.grid_values(kind, bits)[0].astype(np.float32)).cuda()
    codes = torch.randint(0, values.numel(), (outputs, width), generator=generator, device="cuda", dtype=torch.uint8)
    groups = width // group
    scales = (torch.rand(outputs, groups, generator=generator, device="cuda") * 0.01 + 0.001).half()
    zero = (torch.randn(outputs, groups, generator=generator, device="cuda") * 0.02).half() if zeros else None
    from mlkit_b200 import pack

    dense = values.double()[codes.long()] * scales.double().repeat_interleave(group, 1)
    if zeros:
        dense = dense + zero.double().repeat_interleave(group, 1)
    return {"packed": pack(codes, bits), "scales": scales, "values": values, "zeros": zero, "dense": dense,
            "bits": bits, "group": group, "outputs": outputs}


def run(layer, x, kernel="auto", bias=None):
    from mlkit_b200 import kernels

    integer, low = kernels.integer_grid_of(layer["values"])
    out = torch.full((x.shape[0], layer["outputs"]), float("nan"), dtype=x.dtype, device="cuda")
    return kernels.packed_matvec(x, layer["packed"], layer["scales"], layer["values"], layer["zeros"], bias, out,
                                 group=layer["group"], bits=layer["bits"], integer_grid=integer, grid_minimum=low,
                                 kernel=kernel)


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind,bits,group,zeros", FORMS)
def test_every_form_against_64_bits(kind, bits, group, zeros, dtype):
    generator = torch.Generator(device="cuda").manual_seed(3)
    # one k-tile; ragged rows; an odd number of k-tiles; several row groups; K split over a cluster
    for outputs, width in ((16, 128), (30, 256), (1002, 896), (4098, 2048), (72, 4480), (520, 9216)):
        layer = layer_of(kind, bits, group, zeros, outputs, width, seed=outputs)
        for rows in (1, 3, 8):
            x = torch.randn(rows, width, generator=generator, device="cuda").to(dtype)
            bias = torch.randn(outputs, generator=generator, device="cuda").to(dtype) if rows == 3 else None
            expected = x.double() @ layer["dense"].t()
            if bias is not None:
                expected = expected + bias.double()
            assert rel(run(layer, x, bias=bias), expected) <= BOUND[dtype], (outputs, width, rows)


@pytest.mark.parametrize("kind,bits,group,zeros", [("int", 4, 128, False), ("int", 4, 32, True), ("int", 8, 128, False),
                                                   ("nf4", 4, 64, False), ("codebook3", 3, 64, False)])
def test_bf16_range(kind, bits, group, zeros):
    """Magnitudes fp16 cannot hold, rows of very different size, and channels far apart within a row."""
    generator = torch.Generator(device="cuda").manual_seed(5)
    layer = layer_of(kind, bits, group, zeros, 200, 1024)
    x = torch.randn(5, 1024, generator=generator, device="cuda")
    x[0] *= 1e30
    x[1] *= 1e-30
    x[2] *= torch.logspace(-6, 6, 1024, device="cuda")
    x[3] = 0
    x = x.bfloat16()
    expected, got = x.double() @ layer["dense"].t(), run(layer, x)
    for row in (0, 1, 2, 4):
        assert rel(got[row], expected[row]) <= BOUND[torch.bfloat16], row
    assert torch.equal(got[3], torch.zeros_like(got[3]))


@pytest.mark.parametrize("bits,group", [(4, 64), (4, 128), (3, 64), (3, 128)])
def test_bf16_tables_of_far_apart_levels(bits, group):
    """Levels down to 2^-36 of the largest, in weight rows that hold levels of one size each.  A level is held to 22
    bits or to 2^-39 of the largest: at 2^-30 that is 2^-9 of it, beside the output's own 2^-8."""
    from mlkit_b200 import pack

    generator = torch.Generator(device="cuda").manual_seed(9)
    layer = layer_of("codebook3" if bits == 3 else "nf4", bits, group, False, 64, 1024)
    sizes = 2.0 ** torch.tensor([0, -10, -20, -24, -25, -27, -30, -36], device="cuda")
    values = torch.cat((1.3 * sizes, sizes)) if bits == 4 else 1.3 * sizes
    pairs = torch.randint(0, 2, (64, 1024), generator=generator, device="cuda") * (8 if bits == 4 else 0)
    codes = (torch.arange(64, device="cuda")[:, None] % 8 + pairs).to(torch.uint8)
    layer.update(values=values, packed=pack(codes, bits))
    layer["dense"] = values.double()[codes.long()] * layer["scales"].double().repeat_interleave(group, 1)
    x = torch.rand(3, 1024, generator=generator, device="cuda").bfloat16()
    got, expected = run(layer, x), x.double() @ layer["dense"].t()
    for size in range(7):
        assert rel(got[:, size::8], expected[:, size::8]) <= BOUND[torch.bfloat16] + 2.0**-9, float(sizes[size])
    assert rel(got[:, 7::8], expected[:, 7::8]) <= 2.0**-2     # 2^-36 is held to an eighth of itself


@pytest.mark.parametrize("width", [1024, 9216])
@pytest.mark.parametrize("kind,bits,group,zeros", [("int", 4, 128, False), ("int", 4, 64, True), ("int", 3, 128, False),
                                                   ("nf4", 4, 64, False)])
def test_bf16_infinities_and_nans(kind, bits, group, zeros, width):
    """Rows with an infinity or a NaN answer what the general kernel answers; the other rows are untouched."""
    generator = torch.Generator(device="cuda").manual_seed(6)
    layer = layer_of(kind, bits, group, zeros, 100, width)
    x = torch.randn(4, width, generator=generator, device="cuda").bfloat16()
    clean = run(layer, x)
    dirty = x.clone()
    dirty[0, 77] = float("inf")
    dirty[1, width - 1] = float("-inf")
    dirty[1, 5] = float("nan")
    dirty[3, 200], dirty[3, 300] = float("inf"), float("-inf")
    got, general = run(layer, dirty), run(layer, dirty, kernel="scalar")
    assert torch.equal(got[2], clean[2])
    for row in (0, 1, 3):
        assert torch.equal(got[row].isnan(), general[row].isnan())
        finite = ~general[row].isnan()
        assert torch.equal(got[row][finite], general[row][finite])
    assert got[0].isinf().any()


@pytest.mark.parametrize("width", [128, 1024, 9216])
@pytest.mark.parametrize("kind,bits,group,zeros", [("int", 4, 64, False), ("int", 4, 32, False), ("int", 4, 128, True),
                                                   ("int", 4, 64, True), ("int", 4, 32, True), ("nf4", 4, 64, False)])
def test_fp16_infinities_and_nans(kind, bits, group, zeros, width):
    """The same with fp16, in the forms that once took kernels of whole weights: an infinity stays a signed infinity."""
    generator = torch.Generator(device="cuda").manual_seed(6)
    layer = layer_of(kind, bits, group, zeros, 100, width)
    x = torch.randn(8, width, generator=generator, device="cuda").half()
    clean = run(layer, x)
    dirty = x.clone()
    dirty[0, 77] = float("inf")
    dirty[1, width - 1], dirty[1, 5] = float("-inf"), float("nan")
    dirty[3, 20], dirty[3, 30] = float("inf"), float("-inf")
    dirty[7, 0] = float("-inf")
    got, general = run(layer, dirty), run(layer, dirty, kernel="scalar")
    assert torch.equal(got[[2, 4, 5, 6]], clean[[2, 4, 5, 6]])
    for row in (0, 1, 3, 7):
        assert torch.equal(got[row].isnan(), general[row].isnan())
        finite = ~general[row].isnan()
        assert torch.equal(got[row][finite], general[row][finite])
    assert got[0].isinf().any() and got[7].isinf().any() and not got[7, layer["dense"][:, 0] != 0].isnan().any()


@pytest.mark.parametrize("kind,group", [("int", 64), ("nf4", 64)])
def test_gated_and_rotated_rows_that_are_not_finite(kind, group):
    """Forms that make their activations on load: the gate's product overflows to an infinity, or an input is one."""
    from mlkit_b200 import kernels

    generator = torch.Generator(device="cuda").manual_seed(8)
    layer = layer_of(kind, 4, group, False, 100, 1024)
    integer, low = kernels.integer_grid_of(layer["values"])
    form = dict(group=group, bits=4, integer_grid=integer, grid_minimum=low)
    held = layer["packed"], layer["scales"], layer["values"], None

    def gated(both):
        out = torch.full((both.shape[0], 100), float("nan"), dtype=torch.float16, device="cuda")
        return kernels.packed_matvec(both, *held, None, out, gated=True, **form)

    both = torch.randn(3, 2048, generator=generator, device="cuda").half()
    clean = gated(both)
    both[1, 7], both[1, 1024 + 7] = 600.0, -600.0          # fp16 ends at 65504
    got, weights = gated(both), layer["dense"][:, 7]
    assert torch.equal(got[[0, 2]], clean[[0, 2]])
    assert torch.equal(got[1].isnan(), weights == 0)
    assert torch.equal(got[1][weights != 0].double(), weights[weights != 0].sign() * float("-inf"))

    x = torch.randn(3, 1024, generator=generator, device="cuda").half()
    x[1, 9] = float("inf")
    signs = (torch.randint(0, 2, (1024,), generator=generator, device="cuda") * 2 - 1).to(torch.int8)
    out = torch.empty(3, 100, dtype=torch.float16, device="cuda")
    kernels.packed_matvec_rotated(x, signs, *held, out, **form)
    expected = run(layer, kernels.structured_transform(x, factor=1, power=1024, signs=signs))
    assert torch.equal(out.isnan(), expected.isnan()) and torch.equal(out.nan_to_num(), expected.nan_to_num())


def test_forms_left_to_other_kernels():
    """Layouts outside the streaming kernel still answer, and its explicit choice refuses what it refused."""
    generator = torch.Generator(device="cuda").manual_seed(7)
    for kind, bits, group, zeros, width in (("int", 4, 16, False, 256), ("int", 8, 64, False, 256), ("int", 4, 128, False, 192),
                                            ("int", 3, 128, True, 256), ("int", 4, 96, False, 192)):
        layer = layer_of(kind, bits, group, zeros, 40, width) if width % group == 0 else None
        if layer is None:
            continue
        x = torch.randn(2, width, generator=generator, device="cuda").bfloat16()
        assert rel(run(layer, x), x.double() @ layer["dense"].t()) <= BOUND[torch.bfloat16]
    layer = layer_of("int", 4, 128, False, 32, 256)
    for x, held in ((torch.randn(2, 256, device="cuda").bfloat16(), layer),
                    (torch.randn(2, 256, device="cuda").half(), layer_of("int", 4, 128, True, 32, 256)),
                    (torch.randn(2, 256, device="cuda").half(), layer_of("int", 4, 32, False, 32, 256))):
        with pytest.raises(ValueError):
            run(held, x, kernel="stream")
    # a base address off the 16-byte boundary takes the general kernel
    x = torch.randn(2 * 256 + 1, generator=generator, device="cuda").bfloat16()[1:].view(2, 256)
    assert rel(run(layer, x), x.double() @ layer["dense"].t()) <= BOUND[torch.bfloat16]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("outputs", [32768, 34816, 36864])
def test_wide_layers_of_long_rows(outputs, dtype):
    """K of 32768 is split over clusters of eight CTAs; how many of those the GPU holds decides whether a launch of this
    width needs more visits than it keeps sums for, and such a call takes another kernel."""
    generator = torch.Generator(device="cuda").manual_seed(11)
    width = 32768
    packed = torch.randint(0, 256, (outputs * width // 2,), generator=generator, device="cuda", dtype=torch.uint8)
    scales = (torch.rand(outputs, width // 128, generator=generator, device="cuda") * 0.01 + 0.001).half()
    layer = {"packed": packed, "scales": scales, "values": torch.arange(-8, 8, device="cuda").float(), "zeros": None,
             "bits": 4, "group": 128, "outputs": outputs}
    x = torch.randn(2, width, generator=generator, device="cuda").to(dtype)
    got = run(layer, x)
    for first in (0, outputs - 48):
        part = {**layer, "packed": packed[first * width // 2:(first + 48) * width // 2], "scales": scales[first:first + 48], "outputs": 48}
        assert rel(got[:, first:first + 48], run(part, x, kernel="scalar").double()) <= 2 * BOUND[dtype]
