"""The kernels' short forms of quotients and of the exponential, on the device, against the operations they stand
for: equal bits over every value where the claim is about every value, else over the range they are used in."""
import ctypes as C

import numpy as np
import pytest

from phosphor_b200 import _capi as A

UNORM8, DIV_ZERO, DIV_KNOWN, DIV_GAUSS, EXP_UNIT, EXPF = range(6)
GAUSS_BETA, GAUSS_DENOM = np.float32(1.953), np.float32(0.85815)  # photon_hash.h:88-95


def device(fn, a, b=None):
    a = np.ascontiguousarray(a, np.float32)
    b = np.zeros_like(a) if b is None else np.ascontiguousarray(b, np.float32)
    out = np.empty_like(a)
    vp = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
    A.check(A.load().phx_selftest_math(fn, vp(a), vp(b), vp(out), a.size))
    return out


def equal_bits(got, want):
    return np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.gpu
def test_every_byte_over_255():
    x = np.arange(256, dtype=np.float32)
    assert equal_bits(device(UNORM8, x), x / np.float32(255))


@pytest.mark.gpu
def test_quotients_with_zero_numerators_apart():
    """Signed zeros, subnormals, infinities and NaN in both places, and ordinary values beside them."""
    rng = np.random.default_rng(1)
    tiny = np.float32(1e-45)
    some = np.concatenate([
        np.float32([0, tiny, 3 * tiny, 1.1754942e-38, 1.17549435e-38, 5.4e-20, 1, 0.1, 3, 255, 1e19, 3.4e38, np.inf, np.nan]),
        np.exp2(rng.uniform(-149, 127, 500)).astype(np.float32)])
    some = np.concatenate([some, -some])
    a, b = (v.reshape(-1) for v in np.meshgrid(some, some, indexing="ij"))
    got = device(DIV_ZERO, a, b)
    with np.errstate(all="ignore"):
        want = a / b
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert equal_bits(got[~nan], want[~nan])


@pytest.mark.gpu
def test_quotients_by_known_divisors():
    """What the gather divides: -beta dsq by 2 r^2, dsq < r^2, wherever the quotient is a normal number."""
    rng = np.random.default_rng(2)
    n = 1 << 24
    y = (2 * np.exp2(rng.uniform(-61, 59, n))).astype(np.float32)
    dsq = (np.exp2(-rng.uniform(0, 1, n) ** 3 * 60) * (0.5 * y)).astype(np.float32)
    dsq[::3] = (rng.random(len(dsq[::3])) * 0.5 * y[::3]).astype(np.float32)  # evenly too
    x = -GAUSS_BETA * dsq
    use = (dsq >= 1e-30) & (dsq < 0.5 * y) & (np.abs(x / y) >= 2.0 ** -126)
    assert use.sum() > n // 2
    assert equal_bits(device(DIV_KNOWN, x[use], y[use]), x[use] / y[use])


@pytest.mark.gpu
def test_every_quotient_by_the_kernels_denominator():
    lo, hi = (int(np.float32(v).view(np.uint32)) for v in (2.0 ** -30, 1.5))
    assert device(DIV_GAUSS, np.zeros(1))[0] == 0
    for at in range(lo, hi + 1, 1 << 24):
        x = np.arange(at, min(at + (1 << 24), hi + 1), dtype=np.uint32).view(np.float32)
        assert equal_bits(device(DIV_GAUSS, x), x / GAUSS_DENOM)


@pytest.mark.gpu
def test_exponential_without_range_checks():
    lo, hi = (int(np.float32(v).view(np.uint32)) for v in (2.0 ** -30, 1.0))
    bits = np.arange(lo, hi + 1, 11, dtype=np.uint32)
    t = np.concatenate([-bits.view(np.float32), np.float32([0.0, -0.0, -1.0, -1e-30, -1e-45])])
    assert equal_bits(device(EXP_UNIT, t), device(EXPF, t))
