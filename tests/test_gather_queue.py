"""The queued gather against the warp-cooperative one (the same sums in the same order: equal bits), where
its queue, its cell mask and its exact quotients have their edges: grids of one cell to 255 a side, a
handful of photons, radii that hold no photon, some, and the whole scene, and radii outside the range of
the quotient's short form."""
import numpy as np
import pytest

import phosphor_b200 as P
from phosphor_b200 import _capi as A


def gathered(grid, photons, radius2, coop, w=45, h=37):
    scene = P.SceneData.generate(A.PHX_SCENE_CORNELL, seed=3, width=w, height=h)
    args = P.ArgsList(width=w, height=h, photons_per_round=photons, max_photon_bounces=6, grid_res=grid, seed=9,
                      direct_samples=2)
    with P.Renderer(args) as r:
        r.set_scene(scene)
        t = r.tuning()
        t.gather_coop = coop
        r.set_tuning(t)
        r.round()
        if radius2 is not None:
            flux = r.read("FLUX")
            flux[:, 3] = np.float32(radius2) * np.linspace(0.25, 1.0, len(flux), dtype=np.float32)
            r.write("FLUX", flux)
        r.round()
        return [r.read(b).view(np.uint32) for b in ("FLUX", "PHOTON_WEIGHT", "RADIANCE")], r.read("PHOTON_WEIGHT")


@pytest.mark.gpu
@pytest.mark.parametrize("grid,photons,radius2", [
    (1, 9, None), (1, 700, None), (2, 3000, 0.02), (50, 5, None), (50, 20000, None), (50, 20000, 1.1e-5),
    (50, 20000, 3e-3), (50, 3000, 40.0), (255, 20000, None), (255, 20000, 1e-4), (50, 3000, 1e19), (3, 3000, 1e-6),
])
def test_queued_gather_equals_the_cooperative_one(grid, photons, radius2):
    got, weight = gathered(grid, photons, radius2, 0)
    want, _ = gathered(grid, photons, radius2, 1)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    if radius2 is None or radius2 > 1e-3:
        assert weight.any()
