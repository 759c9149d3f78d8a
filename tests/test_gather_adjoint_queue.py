"""The gather adjoint's queue at its edges: a single pixel, partly filled warps and blocks, and a coarse
grid whose pixels find far more photons than the queue holds, against the oracle's analytic FP64
gradient."""
import numpy as np
import pytest

import oracle as O
import phosphor_b200 as P
from phosphor_b200 import _capi as A

TOL = 1e-3  # of the largest partial: the bound that the float adjoint is held to everywhere


@pytest.mark.gpu
@pytest.mark.parametrize("size,grid", [((1, 1), 4), ((33, 1), 4), ((13, 11), 4), ((13, 11), 40)])
def test_gather_adjoint_matches_the_analytic_gradient(size, grid):
    w, h = size
    scene = P.SceneData.generate(A.PHX_SCENE_CORNELL, seed=3, width=w, height=h, detail=0)
    args = P.ArgsList(width=w, height=h, photons_per_round=1 << 13, max_photon_bounces=6, grid_res=grid, seed=3,
                      direct_samples=4, sppm_alpha=0.7)
    g = np.random.default_rng(5).uniform(0.5, 1.5, w * h * 3).astype(np.float32)
    with P.Renderer(args) as r:
        r.set_scene(scene)
        r.adjoint_forward(2)
        got = r.adjoint_backward(g).astype(np.float64)
    want, _ = O.Oracle(scene).frozen_grad(args.params(), 2, scene.materials(), scene.lights(), g.astype(np.float64))
    scale = np.abs(want).max()
    assert scale > 0
    # a roughness at its clamp (1, all of this scene's) reports 0 by definition: those coordinates have no counterpart
    at_clamp = np.zeros(len(want), bool)
    at_clamp[3:4 * len(scene.materials()):4] = scene.materials()["roughness"] >= 1.0
    assert np.all(got[at_clamp] == 0.0)
    assert np.abs(got - want)[~at_clamp].max() <= TOL * scale
