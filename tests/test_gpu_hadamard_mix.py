"""The tensor-core form of the structured transform (many 16-bit rows, Hadamard factor basis) against a 64-bit one, and
against the factor kernel for what is not finite.

Tolerance: the mix is exact up to fp32 accumulation and the butterflies round in fp32 (a few 2^-24 each), so the one
rounding of the output decides: at most 2^-11 of a value in fp16, 2^-8 in bf16.
"""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
BOUND = {torch.float16: 2.0**-11 * 1.01, torch.bfloat16: 2.0**-8 * 1.01}


def plain(x, signs, factor, power, basis, inverse):
    y = x.double() if inverse or signs is None else x.double() * signs
    span = 1
    while span < power:
        pairs = y.reshape(-1, 2, span)
        y = torch.stack((pairs[:, 0] + pairs[:, 1], pairs[:, 0] - pairs[:, 1]), 1)
        span *= 2
    y = (y / math.sqrt(power)).reshape(-1, factor, power)
    mix = basis.double().cuda()
    y = torch.matmul(mix.t() if inverse else mix, y).reshape(x.shape)
    return y * signs if inverse and signs is not None else y


@pytest.mark.parametrize("width", [36 * 1024, 44 * 1024])
def test_widths_that_stay_with_the_factor_kernel(width):
    """Rows too wide for the shared memory of the tensor-core form, through the public call."""
    import mlkit_b200 as mk
    from mlkit_b200 import transforms

    factor, power, basis = transforms.transform_factor(width)
    assert (factor, power) == (width // 1024, 1024) and transforms._hadamard_basis(width)
    x, signs = torch.randn(96, width, device="cuda"), (torch.randint(0, 2, (width,), device="cuda") * 2 - 1).to(torch.int8)
    for dtype in BOUND:
        for inverse in (False, True):
            expected = plain(x.to(dtype), signs, factor, power, basis, inverse)
            got = mk.rht(x.to(dtype), signs=signs, inverse=inverse)
            assert float((got.double() - expected).norm() / expected.norm()) <= BOUND[dtype]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("width", [12 * 128, 44 * 128, 20 * 256, 36 * 256, 28 * 512, 36 * 512, 12 * 1024, 28 * 1024])
def test_against_64_bits(width, dtype):
    from mlkit_b200 import transforms

    factor, power, basis = transforms.transform_factor(width)
    assert transforms._hadamard_basis(width)
    generator = torch.Generator(device="cuda").manual_seed(width)
    signs = (torch.randint(0, 2, (width,), generator=generator, device="cuda") * 2 - 1).to(torch.int8)
    for rows in (64, 297, 601):    # fewer rows than CTAs, one CTA with a second row, several each
        x = torch.randn(rows, width, generator=generator, device="cuda")
        x[:, ::97] *= 50
        x = x.to(dtype)
        for inverse in (False, True):
            for s in (signs, None):
                got = transforms.structured_transform(x, inverse=inverse, signs=s)
                expected = plain(x, s, factor, power, basis, inverse)
                assert float((got.double() - expected).norm() / expected.norm()) <= BOUND[dtype], (rows, inverse)


def test_row_count_does_not_change_a_row():
    """The same row through either kernel: equal up to the rounding of the output."""
    from mlkit_b200 import kernels, transforms

    x = torch.randn(100, 14336, device="cuda").half()
    many, few = transforms.structured_transform(x), transforms.structured_transform(x[:4])
    assert float((many[:4].float() - few.float()).norm() / few.float().norm()) <= 2.0**-11
    strided = transforms.structured_transform(torch.cat((x, x), 1)[:, 14336:])     # a view is copied first
    assert torch.equal(strided, many)
    in_place = x.clone()
    kernels.structured_transform(in_place, factor=28, power=512, basis=transforms._device_basis(14336, x.device),
                                 out=in_place, hadamard_basis=True)
    assert torch.equal(in_place, many)
    offset = torch.empty(100 * 14336 + 1, device="cuda", dtype=torch.float16)[1:].view(100, 14336).copy_(x)
    assert float((transforms.structured_transform(offset).float() - many.float()).norm() / many.float().norm()) <= 2.0**-11


def test_not_finite_rows():
    from mlkit_b200 import transforms

    x = torch.randn(80, 6144, device="cuda").half()
    clean = transforms.structured_transform(x)
    x[3, 700], x[9, 5], x[9, 6000], x[20, 1] = float("inf"), float("inf"), float("-inf"), float("nan")
    got = transforms.structured_transform(x)
    general = torch.cat([transforms.structured_transform(x[i:i + 8]) for i in range(0, 80, 8)])
    assert torch.equal(got.isnan(), general.isnan()) and torch.equal(got.isinf(), general.isinf())
    assert torch.equal(got[got.isinf()], general[general.isinf()])
    untouched = [i for i in range(80) if i not in (3, 9, 20)]
    assert torch.equal(got[untouched], clean[untouched])


def test_threads_with_factors_of_one_instance():
    """10240 = 20 x 512 and 14336 = 28 x 512 share a kernel instance and need different amounts of shared memory."""
    import threading

    from mlkit_b200 import transforms

    inputs = [torch.randn(64, width, device="cuda").half() for width in (10240, 14336)]
    expected = [transforms.structured_transform(x) for x in inputs]
    failures = []

    def work(index):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(1500):
                    got = transforms.structured_transform(inputs[index])
                torch.cuda.current_stream().synchronize()
            assert torch.equal(got, expected[index])
        except Exception as error:
            failures.append(error)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(index,)) for index in (0, 1, 0, 1)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not failures, failures[0]
