"""Gradients with more parameters than a block's shared memory holds (over 8192: from about 2050 materials on),
where every sum goes straight into the global doubles."""
import ctypes as C
import math

import numpy as np
import pytest

import phosphor_b200 as P
from phosphor_b200 import _capi as A


def scene_of(kind, detail, w, h, n_mat, light_power=None):
    """A generated scene with its material table filled up to n_mat by materials that nothing uses."""
    base = P.SceneData.generate(kind, seed=3, width=w, height=h, detail=detail)
    mats, lights = base.materials(), base.lights().copy()
    if n_mat:
        mats = np.concatenate([mats, np.repeat(mats[-1:], n_mat - len(mats))])
    if light_power is not None:
        for c in "xyz":
            lights["power"][c] = light_power
    sc = A.Scene.from_buffer_copy(base.scene)
    uvt = (A.UvTransformBlock * len(mats))()
    for i in range(base.scene.n_materials):
        C.memmove(C.byref(uvt[i]), C.byref(base.scene.uv_transforms[i]), C.sizeof(A.UvTransformBlock))
    sc.materials, sc.n_materials = C.cast(mats.ctypes.data, C.POINTER(A.Material)), len(mats)
    sc.uv_transforms = uvt
    sc.lights, sc.lum_pref_sum = C.cast(lights.ctypes.data, C.POINTER(A.Light)), None
    return P.SceneData(sc, keep=(base, mats, lights, uvt))


def args_of(w, h, photons, samples):
    return P.ArgsList(width=w, height=h, photons_per_round=photons, max_photon_bounces=8, grid_res=24, seed=3,
                      direct_samples=samples, sppm_alpha=0.7)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,detail", [(A.PHX_SCENE_ATRIUM, 4), (A.PHX_SCENE_CAUSTIC, 24)])
@pytest.mark.parametrize("wavefront", [1, 0])
def test_same_gradient_as_with_few_materials(kind, detail, wavefront):
    """The bound covers the few-material side, which sums up to 1e5 float terms in blocks of 128 threads:
    128 roundings of 2^-24 a block, with room for terms that cancel."""
    w, h = 61, 47
    g = np.random.default_rng(8).standard_normal(w * h * 3).astype(np.float32)
    got = []
    for n_mat in (0, 2100):
        scene = scene_of(kind, detail, w, h, n_mat)
        with P.Renderer(args_of(w, h, 1 << 13, 4)) as r:
            r.set_scene(scene)
            t = r.tuning()
            t.nee_wavefront = t.persistent = wavefront
            r.set_tuning(t)
            r.adjoint_forward(2)
            got.append(r.adjoint_backward(g).astype(np.float64))
    few, many = got
    n = len(scene_of(kind, detail, w, h, 0).materials())
    assert len(many) > 8192
    scale = np.abs(few).max()
    assert scale > 0 and not many[4 * n:4 * 2100].any()
    assert np.abs(many[:4 * n] - few[:4 * n]).max() <= 1e-4 * scale
    assert np.abs(many[4 * 2100:] - few[4 * n:]).max() <= 1e-4 * scale


@pytest.mark.gpu
def test_small_terms_survive_beside_large_ones():
    """The gradient of one light's power over pixels that see it directly and nothing else (a diffuse first hit,
    one sample, no photon) is sum g_p direct_p / power, each term exact for powers of two g and power.  In
    every 32 pixels the first such has g = 1 and the others a g that leaves their terms just under half an ulp of
    the first one's: a float sum over these loses all 31 of them, about 9 ulp, while in double only the
    result's own rounding to float is left."""
    w, h = 64, 48
    power = 256.0
    scene = scene_of(A.PHX_SCENE_ATRIUM, 4, w, h, 2100, power)
    with P.Renderer(args_of(w, h, 64, 1)) as r:
        r.set_scene(scene)
        r.adjoint_forward(1)
        direct = r.read("HP_DIRECT").reshape(-1, 4)[:, 0].astype(np.float64)
        emission = r.read("HP_EMISSION").reshape(-1, 4)
        plain = (emission == (0, 0, 0, 1)).all(1) & (r.read("HP_THROUGHPUT").reshape(-1, 4)[:, :3] == 1).all(1)
        plain &= (r.read("PHOTON_WEIGHT") == 0) & (direct > 0)
        g = np.zeros((w * h, 3), np.float32)
        used = 0
        for j in range(0, w * h, 32):
            lanes = j + np.flatnonzero(plain[j:j + 32])
            if len(lanes) < 2:
                continue
            g[lanes[0], 0] = 1.0
            room = 0.45 * float(np.spacing(np.float32(direct[lanes[0]])))
            for p in lanes[1:]:
                g[p, 0] = 2.0 ** math.floor(math.log2(room / direct[p]))
                used += 1
        assert used > 300
        got = r.adjoint_backward(g.reshape(-1)).astype(np.float64)
    want = math.fsum(g[:, 0].astype(np.float64) * direct) / power
    assert abs(got[4 * 2100] - want) <= 1.01 * 2.0 ** -24 * want
