"""A filter whose result overwrites its image, in page-locked memory, where the upload is still reading while
the host prepares the result buffer (which it does for results of 8 MB and more)."""
import ctypes as C

import numpy as np
import pytest

from phosphor_b200 import _capi as A

W, H = 1103, 701  # 9.3 MB of int32 or float32, 18.6 MB of float64


def vp(a, offset=0):
    return C.c_void_p(a.ctypes.data + offset)


def image(dtype):
    return np.random.default_rng(3).integers(1, 255, size=(H, W, 3)).astype(dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["phx_mean_filter", "phx_median_filter"])
def test_float_result_over_its_int_image(name):
    import torch

    img = image(np.int32)
    want = np.empty((H, W, 3), np.float32)
    A.check(getattr(A.load(), name)(vp(img), vp(want), W, H, 1, None))
    buf = torch.empty(img.size, dtype=torch.int32, pin_memory=True).numpy()
    for _ in range(3):
        buf[:] = img.reshape(-1)
        A.check(getattr(A.load(), name)(vp(buf), vp(buf), W, H, 1, None))
        assert np.array_equal(buf.view(np.uint32), want.view(np.uint32).reshape(-1))


@pytest.mark.gpu
@pytest.mark.parametrize("at", ["front", "back"])
def test_double_result_over_its_byte_image(at):
    import torch

    img = image(np.uint8)
    want = np.empty((H, W, 3), np.float64)
    A.check(A.load().phx_filter_f64(0, vp(img), 1, vp(want), None, W, H, 1, None))
    buf = torch.empty(img.size, dtype=torch.float64, pin_memory=True).numpy()
    off = 0 if at == "front" else buf.nbytes - img.nbytes
    for _ in range(3):
        buf.view(np.uint8)[off:off + img.nbytes] = img.reshape(-1)
        A.check(A.load().phx_filter_f64(0, vp(buf, off), 1, vp(buf), None, W, H, 1, None))
        assert np.array_equal(buf.view(np.uint64), want.view(np.uint64).reshape(-1))
