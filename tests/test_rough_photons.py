"""The photon kernel that searches its microfacet attempts with a cheap test (chosen for mostly rough
scenes) against the one-thread kernel, which computes every attempt: the same photons, bit for bit, at
the roughness where the kernel is chosen and past the clamp, for metals, dielectrics, glass and mixes, and
with one near-mirror among the rough surfaces."""
import numpy as np
import pytest

import phosphor_b200 as P
from phosphor_b200 import _capi as A


def photons(scene, mats, flags):
    args = P.ArgsList(width=32, height=32, photons_per_round=1 << 16, max_photon_bounces=12, grid_res=40, seed=12,
                      direct_samples=1, flags=flags)
    with P.Renderer(args) as r:
        r.set_scene(scene)
        r.set_materials(mats)
        r.round()
        assert r.info().n_photons > 1000
        return [r.read(b).view(np.uint32) for b in ("EMIT_COUNT", "PHOTON_POS", "PHOTON_POWER", "PHOTON_DIR")]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,detail", [(A.PHX_SCENE_CAUSTIC, 40), (A.PHX_SCENE_ATRIUM, 6)])
@pytest.mark.parametrize("roughness", [0.6, 0.85, 1.0, 2.5])
@pytest.mark.parametrize("metallic", [0.0, 0.5, 1.0])
def test_searched_attempts_give_the_same_photons(kind, detail, roughness, metallic):
    scene = P.SceneData.generate(kind, seed=5, width=32, height=32, detail=detail)
    mats = scene.materials().copy()
    mats["roughness"] = np.where(np.arange(len(mats)) == len(mats) - 1, 0.02, 1.2 * roughness).astype(np.float32)
    mats["metallic"][::2] = metallic
    for a, b in zip(photons(scene, mats, 0), photons(scene, mats, A.PHX_F_SIMPLE_TRAVERSAL)):
        assert np.array_equal(a, b)
