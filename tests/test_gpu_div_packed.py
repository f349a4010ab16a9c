"""The packed quotients and roots of the erosion kernels, in the ranges that the kernels test for, against the correctly
rounded ones: a double-precision quotient or root rounded to single precision is the correctly rounded one
(53 >= 2 x 24 + 2 bits)."""
from __future__ import annotations

import pytest

import master_thesis_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    assert t.cuda.is_available(), "a CUDA GPU is required"
    return t


def packed(torch, a, b, amplitude=1.0):
    q, r = torch.empty_like(a), torch.empty_like(a)
    T.check(T.lib().tecto_selftest_packed(a.data_ptr(), b.data_ptr(), amplitude, q.data_ptr(), r.data_ptr(), a.numel(),
                                          torch.cuda.current_stream().cuda_stream), "tecto_selftest_packed")
    return q, r


def floats(torch, g, n, lo, hi):
    """Magnitudes of [2^lo, 2^hi), every exponent alike."""
    e = torch.randint(lo + 127, hi + 127, (n,), device="cuda", generator=g, dtype=torch.int32)
    m = torch.randint(0, 1 << 23, (n,), device="cuda", generator=g, dtype=torch.int32)
    return ((e << 23) | m).view(torch.float32)


def test_roots_of_every_float_of_the_range(torch):
    one = torch.ones(1 << 23, device="cuda")
    for e in range(-100, 64):
        a = (((e + 127) << 23) + torch.arange(1 << 23, device="cuda", dtype=torch.int32)).view(torch.float32)
        assert torch.equal(packed(torch, a, one)[1], a.double().sqrt().float()), f"2^{e}"
    ends = torch.tensor([0.0, 2.0 ** 64], device="cuda")
    assert torch.equal(packed(torch, ends, ends + 1)[1], ends.sqrt())


def test_quotients(torch):
    g = torch.Generator(device="cuda").manual_seed(3)
    n = 1 << 24
    for lo, hi in ((-90, 64), (-40, 10), (-3, 3)):
        a = floats(torch, g, n, lo, hi) * (torch.randint(0, 2, (n,), device="cuda", generator=g) * 2 - 1)
        b = floats(torch, g, n, -32, 32)
        a[:4] = torch.tensor([0.0, 2.0 ** -90, -(2.0 ** -90), 2.0 ** 63], device="cuda")
        b[:4] = torch.tensor([2.0 ** -32, 2.0 ** 32, 2.0 ** 32, 2.0 ** -32], device="cuda")
        assert torch.equal(packed(torch, a, b)[0], (a.double() / b.double()).float())


@pytest.mark.parametrize("k", [-16, -9, -1, 1, 16])
def test_quotients_with_the_amplitude_folded_in(torch, k):
    """The thermal march: dividends above 2^-32, a sum of up to eight of them as divisor."""
    g = torch.Generator(device="cuda").manual_seed(k + 20)
    n = 1 << 24
    a = floats(torch, g, n, -32, 29)
    b = torch.clamp(a * (1 + 7 * torch.rand(n, device="cuda", generator=g)), min=2.0 ** -32, max=2.0 ** 32)
    want = 2.0 ** k * (a.double() / b.double()).float()
    assert torch.equal(packed(torch, a, b, 2.0 ** k)[0], want)
