"""The backward pass with the shadow wavefront's recorded samples against the one that traces every NEE
sample itself (the one-thread forms), over the kinds of scene whose recorded form differs: one point
light (one ray per hit point), an area light seen through glass (occluders), lights that draw differently
(samples drawn in order), several lights, and a batch of rounds of which only the last is still in the
buffers."""
import ctypes as C

import numpy as np
import pytest

import phosphor_b200 as P
from phosphor_b200 import _capi as A

# Both forms sum the same float32 terms (up to ~1e5 of one sign and size per partial, in blocks of 128
# threads, then in double) in different orders: 128 roundings of 2^-24 a block, 1e-5, with room for
# terms that cancel.
TOL = 1e-4


def scene_of(kind, detail, extra, w, h):
    base = P.SceneData.generate(kind, seed=4, width=w, height=h, detail=detail)
    if not extra:
        return base
    lights = base.lights().copy()
    for k in extra:
        new = lights[:1].copy()
        new["kind"], new["aux"] = k, np.zeros(1, new["aux"].dtype)
        new["aux"]["x"], new["aux"]["y"] = 0.5, 0.9
        for f, v in (("position", (0.4, 0.9, 0.6, 0)), ("direction", (0.1, -0.9, -0.2, 0)),
                     ("power", (0.8, 0.7, 0.5, 0))):
            for c, x in zip("xyzw", v):
                new[f][c] = x
        lights = np.concatenate([lights, new])
    sc = A.Scene.from_buffer_copy(base.scene)
    sc.lights, sc.n_lights, sc.lum_pref_sum = C.cast(lights.ctypes.data, C.POINTER(A.Light)), len(lights), None
    return P.SceneData(sc, keep=(base, lights))


CASES = {
    "point_light": (A.PHX_SCENE_ATRIUM, 4, (), 4),
    "glass": (A.PHX_SCENE_CAUSTIC, 24, (), 4),
    "glass_few_samples": (A.PHX_SCENE_CAUSTIC, 24, (), 3),
    "area_and_spot": (A.PHX_SCENE_CAUSTIC, 24, (A.PHX_LIGHT_SPOT,), 5),
    "two_points": (A.PHX_SCENE_ATRIUM, 4, (A.PHX_LIGHT_POINT,), 4),
}


def gradients(scene, args, wavefront, rounds, g):
    with P.Renderer(args) as r:
        r.set_scene(scene)
        t = r.tuning()
        t.nee_wavefront = t.persistent = int(wavefront)
        r.set_tuning(t)
        r.adjoint_forward(rounds)
        first = r.adjoint_backward(g)
        again = r.adjoint_backward(2.0 * g) / 2.0  # the buffers hold another round by now
        r.trace_rays(99)                           # and here no recorded one
        last = r.adjoint_backward(g)
        return first.astype(np.float64), again.astype(np.float64), last.astype(np.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("rounds", [1, 3])
def test_recorded_samples_give_the_traced_gradient(name, rounds):
    kind, detail, extra, samples = CASES[name]
    w, h = 61, 47
    scene = scene_of(kind, detail, extra, w, h)
    args = P.ArgsList(width=w, height=h, photons_per_round=1 << 14, max_photon_bounces=9, grid_res=40, seed=6,
                      direct_samples=samples)
    g = np.random.default_rng(8).standard_normal(w * h * 3).astype(np.float32)
    got = gradients(scene, args, True, rounds, g)
    want = gradients(scene, args, False, rounds, g)
    scale = np.abs(want[0]).max()
    assert scale > 0
    for a in got + want[1:]:
        assert np.abs(a - want[0]).max() <= TOL * scale
