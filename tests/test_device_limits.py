"""Contexts on a nearly full device: rounds in flight give way instead of failing the call, or a later one, and
come back when the tuning is set again."""
import contextlib
import ctypes as C

import numpy as np
import pytest

import phosphor_b200 as P
from phosphor_b200 import _capi as A

W, H = 45, 37
HUGE = 1 << 60


@contextlib.contextmanager
def limit(n):
    """At most n more bytes of device memory; yields a function that says how many were taken."""
    lib, left = A.load(), C.c_uint64()

    def taken():
        A.check(lib.phx_selftest_device_limit(0, C.byref(left)))
        A.check(lib.phx_selftest_device_limit(max(left.value, 1), None))
        return n - left.value

    A.check(lib.phx_selftest_device_limit(n, None))
    try:
        yield taken
    finally:
        A.check(lib.phx_selftest_device_limit(0, None))


@contextlib.contextmanager
def renderer(kind=A.PHX_SCENE_CORNELL, detail=0):
    scene = P.SceneData.generate(kind, seed=3, width=W, height=H, detail=detail)
    args = P.ArgsList(width=W, height=H, photons_per_round=4000, max_photon_bounces=6, grid_res=20, seed=9,
                      direct_samples=4)
    with P.Renderer(args) as r:
        r.set_scene(scene)
        yield r


def state(r):
    return [r.read(b).view(np.uint32).copy() for b in ("FLUX", "RADIANCE", "PHOTON_WEIGHT", "PHOTON_POS")]


def set_bytes():
    """Device memory of one round in flight beside the context's own."""
    with renderer() as r, limit(HUGE) as taken:
        assert r.tuning().pipeline_rounds == 4
        r.iterate(4)
        assert taken() % 3 == 0
        return taken() // 3


@pytest.mark.gpu
@pytest.mark.parametrize("room,kept", [(3.5, 3), (2.5, 1), (1.5, 1), (0.5, 0)])
def test_rounds_in_flight_fit_the_room(room, kept):
    one = set_bytes()
    with renderer() as r:
        r.iterate(11)
        want = state(r)
    with renderer() as r:
        with limit(int(room * one)) as taken:
            for n in (1, 4, 6):
                r.iterate(n)
            assert taken() == kept * one
        for a, b in zip(state(r), want):
            assert np.array_equal(a, b)
        # the room is back: the tuning, set again, takes all its sets
        with limit(HUGE) as taken:
            r.set_tuning(r.tuning())
            r.iterate(4)
            assert taken() == (3 - kept) * one


@pytest.mark.gpu
def test_later_calls_take_the_sets_memory():
    one = set_bytes()

    def calls(r):
        r.iterate(4)
        img = r.image()
        out = [np.ascontiguousarray(img).view(np.uint32)]
        r.iterate(5)
        out += state(r)
        out.append(r.adjoint_forward(1).view(np.uint32))
        return out, r.adjoint_backward(np.ones(W * H * 3, np.float32))

    with renderer() as r:
        want, grad = calls(r)
    with renderer() as r, limit(3 * one + 1000):
        got, grad2 = calls(r)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert np.abs(grad2 - grad).max() <= 1e-5 * np.abs(grad).max()


@pytest.mark.gpu
@pytest.mark.parametrize("start", [4, 2])
@pytest.mark.parametrize("room,most", [(3.5, 4), (1.5, 2), (0.5, 1)])
def test_autotune_keeps_to_groups_that_fit(start, room, most):
    """The state that the tuner keeps aside (36 bytes a pixel) has its own room here."""
    one = set_bytes()
    with renderer() as r:
        t = r.tuning()
        t.pipeline_rounds = start
        r.set_tuning(t)
        with limit(int(room * one) + 40 * W * H) as taken:
            chosen = r.autotune(4)
            assert chosen.pipeline_rounds <= most
            r.iterate(4)
            assert taken() <= (most - 1) * one  # and the state kept aside is back


@pytest.mark.gpu
@pytest.mark.parametrize("concurrent", [0, 1])
def test_autotune_leaves_what_is_no_choice(concurrent):
    """Groups of two are captured the same with and without concurrent_passes, so no trial times it."""
    with renderer() as r:
        t = r.tuning()
        t.concurrent_passes = concurrent
        r.set_tuning(t)
        with limit(set_bytes_of(r) + 40 * W * H):
            for _ in range(3):
                chosen = r.autotune(2)
                assert chosen.pipeline_rounds <= 2 and chosen.concurrent_passes == concurrent


def set_bytes_of(r):
    with limit(HUGE) as taken:
        r.iterate(2)
        return taken()


@pytest.mark.gpu
def test_forward_pass_without_room_for_the_backward_pass():
    """A forward pass needs no photon powers: it renders without them, the backward pass that finds no room
    says so, and one that finds it gives the gradient."""
    g = np.random.default_rng(1).standard_normal(W * H * 3).astype(np.float32)
    with renderer() as r, limit(HUGE) as taken:
        before = taken()
        want = r.adjoint_forward(2).copy()
        forward = taken() - before
        grad = r.adjoint_backward(g)
    slots = 16 * 4000 * 6  # photons per round, bounces
    with renderer() as r:
        with limit(forward - slots) as taken:
            got = r.adjoint_forward(2)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
            assert taken() == forward - slots
            with pytest.raises(A.PhxError) as e:
                r.adjoint_backward(g)
            assert e.value.code == A.PHX_E_OOM
        for _ in range(2):
            assert np.abs(r.adjoint_backward(g) - grad).max() <= 1e-5 * np.abs(grad).max()
