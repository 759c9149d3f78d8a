"""The traversal tree's own box margin (csrc/bvh_margin.hpp): renders equal those of the reference's tree,
whose boxes keep the reference's 1e-3, bit for bit — meshes finer and coarser than the margin, scenes off
the origin, far cameras, every light kind, and lights moved away after set-up."""
import ctypes as C

import numpy as np
import pytest

import phosphor_b200 as P
from phosphor_b200 import _capi as A


def edited(kind, detail, w, h, shift=0.0, back=0.0, light=None):
    """A generated scene moved by `shift` along every axis, its camera pulled `back`, `light` added."""
    base = P.SceneData.generate(kind, seed=2, width=w, height=h, detail=detail)
    tris = base.triangles().copy()
    etris = np.ctypeslib.as_array(base.scene.emissive_triangles, shape=(base.scene.n_emissive_triangles,)).copy() \
        if base.scene.n_emissive_triangles else np.zeros(0, tris.dtype)
    lights = base.lights().copy()
    if light is not None:
        new = lights[:1].copy()
        new["kind"], new["aux"] = light, np.zeros(1, new["aux"].dtype)
        new["aux"]["x"], new["aux"]["y"] = 0.4, 0.7
        for f, v in (("position", (0.5, 0.9, 0.5, 0)), ("direction", (0.1, -0.9, -0.2, 0)),
                     ("tangent", (1, 0, 0, 0)), ("bitangent", (0, 0, 1, 0)), ("power", (1, 1, 1, 0))):
            for c, x in zip("xyzw", v):
                new[f][c] = x
        lights = np.concatenate([lights, new])
    for a in (tris, etris):
        for v in ("v0", "v1", "v2"):
            for c in "xyz":
                a[v][c] += np.float32(shift)
    for c in "xyz":
        lights["position"][c] += np.float32(shift)
    sc = A.Scene.from_buffer_copy(base.scene)
    sc.triangles = C.cast(tris.ctypes.data, C.POINTER(A.Triangle))
    if len(etris):
        sc.emissive_triangles = C.cast(etris.ctypes.data, C.POINTER(A.Triangle))
    sc.lights, sc.n_lights, sc.lum_pref_sum = C.cast(lights.ctypes.data, C.POINTER(A.Light)), len(lights), None
    cam = sc.camera
    for f in ("position", "lower_left_corner"):
        for c in "xyz":
            v = getattr(cam, f)
            setattr(v, c, getattr(v, c) + shift + (back if c == "z" else 0.0))
    return P.SceneData(sc, keep=(base, tris, etris, lights)), lights


def state(r):
    return [r.read(b).view(np.uint32) for b in ("RADIANCE", "FLUX", "PHOTON_POS", "PHOTON_DIR")]


CASES = {
    "water_256": dict(kind=A.PHX_SCENE_CAUSTIC, detail=256),      # triangles of 4 margins
    "water_700": dict(kind=A.PHX_SCENE_CAUSTIC, detail=700),      # triangles of about one margin
    "water_48": dict(kind=A.PHX_SCENE_CAUSTIC, detail=48),        # the margin is the reference's
    "cornell": dict(kind=A.PHX_SCENE_CORNELL, detail=0),          # two triangles a wall
    "shifted": dict(kind=A.PHX_SCENE_CAUSTIC, detail=200, shift=40.0),
    "far_camera": dict(kind=A.PHX_SCENE_CAUSTIC, detail=200, back=30.0),
    "spot": dict(kind=A.PHX_SCENE_CAUSTIC, detail=128, light=A.PHX_LIGHT_SPOT),
    "directional": dict(kind=A.PHX_SCENE_CAUSTIC, detail=128, light=A.PHX_LIGHT_DIRECTIONAL),
    "atrium": dict(kind=A.PHX_SCENE_ATRIUM, detail=24),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("extra", [0, A.PHX_F_BINARY_BVH, A.PHX_F_HOST_BVH])
def test_renders_equal_the_reference_tree(name, extra):
    w, h = 120, 90
    scene, _ = edited(w=w, h=h, **CASES[name])
    got = []
    for flags in (extra, A.PHX_F_REFERENCE_BVH):
        args = P.ArgsList(width=w, height=h, photons_per_round=1 << 16, max_photon_bounces=12, grid_res=50, seed=5,
                          direct_samples=4, flags=flags)
        with P.Renderer(args) as r:
            r.set_scene(scene)
            r.iterate(2)
            assert r.info().stack_overflows == 0
            got.append(state(r))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [0, A.PHX_F_BINARY_BVH])
def test_a_light_moved_away_keeps_the_result(extra):
    w, h = 64, 48
    scene, lights = edited(A.PHX_SCENE_CAUSTIC, 200, w, h, light=A.PHX_LIGHT_POINT)
    far = lights.copy()
    far["position"]["y"][1] = 500.0
    far["power"]["x"][1] = far["power"]["y"][1] = far["power"]["z"][1] = 3.0
    got = []
    for flags in (extra, A.PHX_F_REFERENCE_BVH):
        args = P.ArgsList(width=w, height=h, photons_per_round=1 << 15, max_photon_bounces=12, grid_res=50, seed=5,
                          direct_samples=4, flags=flags)
        with P.Renderer(args) as r:
            r.set_scene(scene)
            r.iterate(1)
            first = state(r)
            r.set_lights(far)
            r.iterate(2)
            got.append(first + state(r))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
