"""Every form of the denoise filters against oracle/filters.py, bit for bit: 8-bit images (which go up as they
are), int32 images, the float64 result of the Python functions and the float32 one of the C entry points, with
windows inside and past the shared-memory tile (k = 8), odd sizes, and a result large enough that its pages are
prepared by several threads (8 MB)."""
import ctypes as C

import numpy as np
import pytest

from oracle import filters as F
from phosphor_b200 import _capi as A
from phosphor_b200 import denoise as D

WINDOWS = {"mean": (0, 1, 2, 8, 9), "median": (0, 1, 2), "weighted": (1, 2, 8, 12)}


def image(shape, dtype, seed=0):
    rng = np.random.default_rng(seed)
    if dtype == np.uint8:
        return rng.integers(0, 256, size=shape + (3,)).astype(np.uint8)
    return rng.integers(-300, 70000, size=shape + (3,)).astype(dtype)


def oracle(name, img, k):
    if name == "mean":
        return F.mean_filter(img, k)
    if name == "median":
        return F.median_filter(img, k)
    return F.weighted_filter(img, D.gaussian_weights(k, 2), k)


def python_form(name, img, k):
    if name == "mean":
        return D.mean_filter_gpu(img, k)
    if name == "median":
        return D.median_filter_gpu(img, k)
    return D.gaussian_filter_gpu(img, k, 2)


def float_form(name, img, k):
    h, w, _ = img.shape
    out = np.full(img.shape, np.nan, np.float32)
    args = [img.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)]
    if name == "weighted":
        wt = np.ascontiguousarray(D.gaussian_weights(k, 2), np.float32)
        args.append(wt.ctypes.data_as(C.c_void_p))
    A.check(getattr(A.load(), f"phx_{name}_filter")(*args, w, h, k, None))
    return out


def same(got, want):
    """Equal bits as float32, and nothing that float32 does not hold."""
    assert np.array_equal(np.float32(got).view(np.uint32), np.float32(want).view(np.uint32))
    assert np.array_equal(np.float32(got).astype(got.dtype), got)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1), (1, 40), (33, 1), (7, 95), (67, 41)])
@pytest.mark.parametrize("name", list(WINDOWS))
def test_byte_images(name, shape):
    img = image(shape, np.uint8, seed=sum(shape))
    for k in WINDOWS[name]:
        got = python_form(name, img, k)
        assert got.dtype == np.float64
        same(got, oracle(name, img.astype(np.int32), k))


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(WINDOWS))
def test_views_of_byte_images(name):
    """Cropped, mirrored and channel-swapped arrays, which are not contiguous."""
    img = image((50, 61), np.uint8, seed=5)
    for view in (img[3:40, 5:50], img[::-1, ::2], img[:, :, ::-1]):
        same(python_form(name, view, 1), oracle(name, np.ascontiguousarray(view).astype(np.int32), 1))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1), (29, 83), (67, 41)])
@pytest.mark.parametrize("name", list(WINDOWS))
def test_float_results(name, shape):
    img = image(shape, np.int32, seed=sum(shape))
    for k in WINDOWS[name]:
        same(float_form(name, img, k), oracle(name, img, k))


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(WINDOWS))
def test_large_results(name):
    img = image((701, 1103), np.uint8, seed=9)  # 18.6 MB of float64, 9.3 MB of float32
    want = oracle(name, img.astype(np.int32), 1)
    same(python_form(name, img, 1), want)
    same(float_form(name, img.astype(np.int32), 1), want)
