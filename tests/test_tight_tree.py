"""The traversal tree with the margin that contexts build theirs with (csrc/bvh_margin.hpp): its structure and its
boxes (CPU), and the GPU build's equality with the host's, array for array."""
import ctypes as C

import numpy as np
import pytest

import phosphor_b200 as P
import test_bvh_build as T
from phosphor_b200 import _capi as A
from phosphor_b200 import renderer as R


def margin(scene, reach):
    """box_margin of every triangle, in its float32 operations."""
    v = scene.triangle_vertices().astype(np.float32)
    e2 = np.zeros(len(v), np.float32)
    for k in range(3):
        d = v[:, (k + 1) % 3] - v[:, k]
        e2 = np.maximum(e2, (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
    unit = np.float32(reach) * np.float32(128.0 / 16777216.0)
    m = unit * (np.float32(1) + e2 * np.float32(1e5))
    return np.where(m < np.float32(1e-3), m, np.float32(1e-3)).astype(np.float32)


def reach_of(scene):
    return float(np.abs(scene.triangle_vertices()).max())


def tree(scene, max_leaf, wide, device, reach, monkeypatch):
    """renderer.traversal_bvh with the margin for `reach`."""
    lib = A.load()
    with monkeypatch.context() as m:
        m.setattr(lib, "phx_traversal_bvh_build",
                  lambda tris, n, leaf, w, dev, out: lib.phx_selftest_traversal_bvh(tris, n, leaf, w, dev, reach, out))
        return R.traversal_bvh(scene, max_leaf, wide, device)


SCENES = {
    "soup": lambda: T.random_soup(3000, 2),
    "thin": lambda: T.random_soup(3000, 6, scale=2.0, size=0.004),  # margins below 1e-3
    "coincident": lambda: T.coincident_soup(300, 200),
    "water": lambda: P.SceneData.generate(A.PHX_SCENE_CAUSTIC, 1, 64, 64, detail=64),
}


@pytest.mark.parametrize("name", list(SCENES))
@pytest.mark.parametrize("wide,max_leaf", [(0, 1), (1, 1), (1, 4), (0, 16)])
def test_host_tree_structure(name, wide, max_leaf, monkeypatch):
    scene = SCENES[name]()
    reach = reach_of(scene)
    m = margin(scene, reach)
    assert np.all(m > 0) and (name not in ("thin", "water") or m.min() < 5e-4)
    v = scene.triangle_vertices().astype(np.float32)
    boxes = v.min(axis=1) - m[:, None], v.max(axis=1) + m[:, None]
    b = tree(scene, max_leaf, wide, -1, reach, monkeypatch)
    monkeypatch.setattr(T, "expanded_boxes", lambda s: boxes)
    T.check_tree(scene, b, bool(wide), max_leaf)
    if max_leaf == 1 and not wide:  # and no box reaches farther: each leaf's is its triangle's own
        for row in b.nodes:
            for k, r in enumerate(row[12:14].view(np.int32)):
                if r < 0:
                    t = b.leaf_tri[~r & ((1 << T.LEAF_BITS) - 1)]
                    lo = np.array([row[4 * k], row[4 * k + 2], row[8 + 2 * k]])
                    hi = np.array([row[4 * k + 1], row[4 * k + 3], row[9 + 2 * k]])
                    assert np.array_equal(lo, boxes[0][t]) and np.array_equal(hi, boxes[1][t])


@pytest.mark.parametrize("name", list(SCENES))
def test_large_reach_is_the_reference_margin(name, monkeypatch):
    scene = SCENES[name]()
    a, b = tree(scene, 4, 1, -1, 1e6, monkeypatch), R.traversal_bvh(scene, 4, 1, -1)
    assert np.array_equal(a.nodes.view(np.uint32), b.nodes.view(np.uint32))
    assert np.array_equal(a.leaf_tri, b.leaf_tri)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(T.gpu_cases()) + ["thin", "water"])
def test_device_tree_equals_host(name, monkeypatch):
    scene = {**T.gpu_cases(), **SCENES}[name]()
    for wide, max_leaf in ((1, 4), (0, 4), (1, 1), (0, 16)):
        h, d = (tree(scene, max_leaf, wide, dev, reach_of(scene), monkeypatch) for dev in (-1, 0))
        assert (d.root, d.depth, d.wdepth) == (h.root, h.depth, h.wdepth)
        assert np.array_equal(d.nodes.view(np.uint32), h.nodes.view(np.uint32))
        assert np.array_equal(d.trirec.view(np.uint32), h.trirec.view(np.uint32))
        assert np.array_equal(d.leaf_tri, h.leaf_tri)
