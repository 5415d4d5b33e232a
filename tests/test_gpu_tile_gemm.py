"""The tensor-core GEMM over packed weights, for every codec form and both activation types, against a 64-bit product
with the weight as the reference reconstructs it (rounded to the activation type); and the routes that lead to it.

Tolerance: the weight is that rounded one bit for bit and products are added in fp32, so the one rounding of the result
decides: at most 2^-11 of a value in fp16, 2^-8 in bf16 (in the norm over a result, whose fp32 errors are far smaller).
"""

import pytest
import torch
from torch.nn import functional

from tests.test_gpu_stream_forms import layer_of, rel

pytestmark = pytest.mark.gpu
BOUND = {torch.float16: 2.0**-11 * 1.01, torch.bfloat16: 2.0**-8 * 1.01}
FORMS = [("int", b, 128, False) for b in range(2, 9)] + [("int", 4, 64, False), ("int", 4, 32, False)] + \
        [("int", 4, 128, True), ("int", 4, 32, True), ("int", 8, 64, True), ("int", 3, 32, True)] + \
        [("nf4", 4, 64, False), ("codebook3", 3, 32, False)]
# a layer of one tile; a ragged second tile; odd N; many blocks of K (tiles cut many times); many tiles of two blocks
SHAPES = [(30, 128), (300, 1024), (1002, 896), (128, 14336), (19999, 256)]


def run(layer, x, bias=None):
    from mlkit_b200 import kernels

    integer, low = kernels.integer_grid_of(layer["values"])
    out = torch.full((x.shape[0], layer["outputs"]), float("nan"), dtype=x.dtype, device="cuda")
    return kernels.packed_tile_gemm(x, layer["packed"], layer["scales"], layer["values"], layer["zeros"], bias, out,
                                    group=layer["group"], bits=layer["bits"], integer_grid=integer, grid_minimum=low)


@pytest.fixture(autouse=True)
def no_expired_wait():
    yield
    from mlkit_b200 import kernels

    assert kernels.gemm_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind,bits,group,zeros", FORMS)
def test_against_64_bits(kind, bits, group, zeros, dtype):
    generator = torch.Generator(device="cuda").manual_seed(5)
    for outputs, width in SHAPES:
        layer = layer_of(kind, bits, group, zeros, outputs, width, seed=outputs)
        dense = layer["dense"].float().to(dtype)
        for rows in (1, 16, 17, 129, 256, 257, 700):
            if rows * outputs > 6_000_000:
                continue
            x = torch.randn(rows, width, generator=generator, device="cuda").to(dtype)
            bias = torch.randn(outputs, generator=generator, device="cuda").to(dtype) if rows % 2 else None
            got = run(layer, x, bias)
            expected = x.double() @ dense.double().t()
            if bias is not None:
                expected = expected + bias.double()
            assert rel(got, expected) <= BOUND[dtype], (outputs, width, rows)
            assert torch.equal(got, run(layer, x, bias))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind,bits,group,zeros", FORMS)
def test_unit_rows_return_the_reconstruction(kind, bits, group, zeros, dtype):
    from mlkit_b200 import kernels

    layer = layer_of(kind, bits, group, zeros, 300, 256)
    weight, _ = kernels.dequantize(layer["packed"], layer["scales"], layer["values"], layer["zeros"], shape=(300, 256),
                                   group=group, bits=bits, dtype=dtype)
    assert torch.equal(run(layer, torch.eye(256, dtype=dtype, device="cuda")).t(), weight)


@pytest.mark.parametrize("group,zeros", [(128, False), (128, True), (64, True), (32, False)])
def test_scales_off_a_word_boundary(group, zeros):
    # an odd number of scales per row, and scales that start on an odd half word
    for outputs, width in ((7, 128), (129, 384), (200, 640)):
        layer = layer_of("int", 4, group, zeros, outputs, width, seed=width)
        x = torch.randn(33, width, device="cuda").half()
        plain = run(layer, x)
        held = torch.empty(layer["scales"].numel() + 1, dtype=torch.float16, device="cuda")
        held[1:] = layer["scales"].flatten()
        assert rel(plain, x.double() @ layer["dense"].float().half().double().t()) <= BOUND[torch.float16]
        assert torch.equal(run({**layer, "scales": held[1:].view_as(layer["scales"])}, x), plain)


def test_infinities_and_nan_follow_the_library():
    layer = layer_of("int", 4, 128, False, 256, 512)
    dense = layer["dense"].float().half()
    x = torch.randn(40, 512, device="cuda").half()
    x[3, 7], x[5, 9], x[30, 100] = float("inf"), float("nan"), -float("inf")
    got, expected = run(layer, x), functional.linear(x, dense)
    assert torch.equal(got.isnan(), expected.isnan()) and torch.equal(got.isposinf(), expected.isposinf())
    assert torch.equal(got.isneginf(), expected.isneginf())


def test_refusals():
    layer = layer_of("int", 4, 64, False, 64, 192)
    with pytest.raises(ValueError):       # K not a multiple of 128
        run(layer, torch.randn(20, 192, device="cuda").half())
    layer = layer_of("int", 4, 16, False, 64, 256)
    with pytest.raises(ValueError):       # 16 codes per scale
        run(layer, torch.randn(20, 256, device="cuda").half())
    layer = layer_of("int", 4, 64, False, 64, 256)
    with pytest.raises(ValueError):
        run(layer, torch.randn(20, 256, device="cuda"))
    with pytest.raises(ValueError):       # activations off a 16-byte boundary
        run(layer, torch.randn(20 * 256 + 1, device="cuda").half()[1:].view(20, 256))


def packed_linear(outputs, width, dtype, cache=False, bias=False):
    import mlkit_b200 as mk

    torch.manual_seed(outputs)
    linear = torch.nn.Linear(width, outputs, bias=bias, device="cuda", dtype=dtype)
    return mk.PackedLinear(linear, mk.int(4)(linear.weight.detach().float(), mk.Ctx("layer", device="cuda")), cache_dense=cache)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("cache", [False, True])
def test_packed_linear_routes(cache, dtype):
    for rows in (9, 16, 17, 32, 33, 128, 129, 512, 513, 1100):
        module = packed_linear(2048, 2048, dtype, cache)
        dense = packed_linear(2048, 2048, dtype).weight.double()
        x = torch.randn(rows, 2048, device="cuda").to(dtype)
        # the matvec's chunks round table levels to fp16 too: three roundings
        bound = 3 * 2.0**-11 if dtype == torch.float16 else BOUND[dtype]
        assert rel(module(x), x.double() @ dense.t()) <= bound, rows
        odd = torch.empty(x.numel() + 1, dtype=dtype, device="cuda")[1:].view_as(x).copy_(x)
        assert rel(module(odd), x.double() @ dense.t()) <= bound, rows


def test_calls_that_see_more_than_values_keep_the_dense_route():
    from torch.autograd import forward_ad

    module = packed_linear(1024, 4096, torch.bfloat16)
    weight = module.weight
    x, tangent = torch.randn(2, 64, 4096, device="cuda").bfloat16()
    assert torch.equal(torch.func.vmap(module)(torch.stack((x, tangent)).unsqueeze(1))[:, 0],
                       torch.func.vmap(lambda v: functional.linear(v, weight))(torch.stack((x, tangent)).unsqueeze(1))[:, 0])
    with forward_ad.dual_level():
        out = forward_ad.unpack_dual(module(forward_ad.make_dual(x, tangent)))
        assert torch.equal(out.tangent, functional.linear(tangent, weight))
    with torch.autocast("cuda", dtype=torch.float16):
        assert module(x).dtype == torch.float16
    assert module(x.requires_grad_()).requires_grad
    with pytest.raises(RuntimeError):       # a bias of another type
        packed_linear(1024, 4096, torch.float32, bias=True)(x.detach())


@pytest.mark.parametrize("bits", [2, 3, 5, 6, 7, 8])
def test_few_rows_of_integer_grids_keep_what_the_matvec_gives(bits):
    """17 to 32 fp16 rows of these grids run as matvec launches, which round no weight: every row is, bit for bit, what
    the matvec gives for it."""
    import mlkit_b200 as mk

    torch.manual_seed(bits)
    linear = torch.nn.Linear(2048, 2048, device="cuda", dtype=torch.float16)
    module = mk.PackedLinear(linear, mk.int(bits)(linear.weight.detach().float(), mk.Ctx("layer", device="cuda")))
    x = torch.randn(32, 2048, device="cuda").half()
    for rows in (17, 24, 32):
        assert torch.equal(module(x[:rows]), torch.cat([module(part) for part in x[:rows].split(8)]))
