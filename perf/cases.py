"""The work that programs built on this package have it do, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes what such a program holds before the call (a
renderer with its scene set, a batch, a parameter vector, an image), `run` is one pass through the
public entry points, `work` what one pass cannot do without, `exact` its result in 64 bits where
plain numpy can give it (a render's random walk has no such value).

Operations:

* render   progressive rounds of one scene followed by its image: `graph` replays captured rounds
           (Renderer.run), `passes` is the per-pass form with its two host reads per round
           (Renderer.run(graph=False)), `seeded` takes each round's seed from the host and shows the
           8-bit image after it (an interactive viewer);
* batch    many small uneven scenes advanced together, every image read back (a dataset or a sweep);
* inverse  one optimisation step: forward render, loss, backward pass to the parameters' gradient;
* denoise  one filter of the denoiser's menu on a finished 8-bit image.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import phosphor_b200 as P
from phosphor_b200 import _capi as A
from phosphor_b200 import denoise
from phosphor_b200.adjoint import ParamTable, render

KINDS = {"cornell": A.PHX_SCENE_CORNELL, "caustic": A.PHX_SCENE_CAUSTIC, "atrium": A.PHX_SCENE_ATRIUM}
# photon path length limit and photon grid of each scene kind's workload
DEPTH = {"cornell": 8, "caustic": 12, "atrium": 16}
GRID = {"cornell": 50, "caustic": 50, "atrium": 64}
# photons stored per photon emitted, about
STORED = {"cornell": 1.8, "caustic": 1.6, "atrium": 0.16}


def _render(name, scene, width, height, photons, rounds, form="graph", detail=0, samples=16, maps=False, spot=False):
    return {"name": name, "op": "render", "scene": scene, "detail": detail, "width": width, "height": height,
            "photons": photons, "rounds": rounds, "form": form, "samples": samples, "maps": maps, "spot": spot}


def listed():
    return [
        # an interactive view of the smallest size: one round, then the 8-bit image, for every seed
        _render("viewer_cornell_64", "cornell", 64, 64, 1 << 14, 1, form="seeded"),
        # the empty box at its workload's size: few triangles, many stored photons
        _render("cornell_512", "cornell", 512, 512, 1 << 18, 4),
        # the headline workload: glass over a diffuse floor, a long chain of crossings per shadow ray
        _render("caustic_1024", "caustic", 1024, 1024, 1 << 20, 4),
        # the largest workload: opaque metal and dielectric under a point light and a sky
        _render("atrium_1080p", "atrium", 1920, 1080, 1 << 22, 2),
        # a small odd-sized glass scene driven pass by pass, with few direct-lighting samples
        _render("passes_caustic_333x251", "caustic", 333, 251, 50001, 2, form="passes", detail=48, samples=5),
        # an asset as glTF files bring them: base colour, metal-rough and normal maps on every material
        _render("textured_atrium_640x361", "atrium", 640, 361, 300007, 3, detail=24, maps=True),
        # an area light beside a spot light: the samples' random draws then differ by light
        _render("two_lights_caustic_400", "caustic", 400, 400, 1 << 18, 3, detail=128, samples=8, spot=True),
        # sixteen small uneven scenes advanced together, one launch per stage
        {"name": "batch_16_small", "op": "batch", "scenes": 16, "side": 64, "photons": 1 << 16, "mix": 7,
         "rounds": 8},
        # one step of the inverse-rendering workload: 131 parameters of the atrium
        {"name": "inverse_atrium_512", "op": "inverse", "scene": "atrium", "detail": 0, "width": 512, "height": 512,
         "photons": 1 << 20, "samples": 16, "rounds": 1},
        # a small fit through glass over two rounds, odd sizes
        {"name": "inverse_caustic_97x65", "op": "inverse", "scene": "caustic", "detail": 32, "width": 97, "height": 65,
         "photons": 20011, "samples": 8, "rounds": 2},
        # the heaviest filter of the denoiser's menu on a full-HD image
        {"name": "median5_1080p", "op": "denoise", "filter": "median", "k": 2, "sd": 1.0, "width": 1920,
         "height": 1080},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["render"] * 6 + ["batch", "inverse", "inverse", "denoise"])
    if op == "denoise":
        side = _log(rng, 100, 1500)
        kind = rng.choice(["mean", "median", "gaussian"])
        return {"op": op, "filter": kind, "k": rng.choice([1, 2]), "sd": rng.choice([1.0, 2.0]),
                "width": side + rng.randrange(64), "height": max(16, int(side * rng.uniform(0.5, 0.95)))}
    if op == "batch":
        return {"op": op, "scenes": rng.randrange(4, 17), "side": rng.choice([48, 64, 96]),
                "photons": _log(rng, 1 << 14, 1 << 16), "mix": rng.randrange(1 << 16), "rounds": rng.randrange(2, 9)}
    scene = rng.choice(["cornell", "caustic", "atrium"])
    detail = {"cornell": 0, "caustic": _log(rng, 16, 256), "atrium": _log(rng, 4, 64)}[scene]
    if op == "inverse":
        side = _log(rng, 40, 480)
        return {"op": op, "scene": scene, "detail": detail, "width": side + rng.randrange(32),
                "height": max(24, int(side * rng.uniform(0.5, 1.0))), "photons": _log(rng, 1 << 13, 1 << 19),
                "samples": rng.choice([4, 8, 16]), "rounds": rng.choice([1, 2])}
    side, photons = _log(rng, 48, 1000), _log(rng, 1 << 13, 1 << 20)
    c = _render("", scene, side + rng.randrange(48), max(32, int(side * rng.uniform(0.5, 1.0))), photons,
                rng.randrange(1, 5), rng.choice(["graph", "graph", "passes", "seeded"]), detail,
                rng.choice([1, 3, 4, 8, 16]), rng.random() < 0.25, rng.random() < 0.25)
    del c["name"]
    return c


def _maps(scene, seed):
    """The scene with texture coordinates and base colour, metal-rough and normal maps."""
    rng = np.random.default_rng(seed)
    tris, mats = scene.triangles().copy(), scene.materials().copy()
    for i in "012":
        v = tris["v" + i]
        tris["uv" + i]["x"] = v["x"] * 0.37 + v["z"] * 0.11
        tris["uv" + i]["y"] = v["y"] * 0.29 + v["z"] * 0.23
    atlas, metas = [], []
    for w, h, lo, hi in ((256, 256, (60, 60, 60), (255, 255, 255)), (128, 96, (200, 40, 0), (255, 255, 255)),
                         (200, 150, (112, 112, 230), (144, 144, 255))):
        metas.append(A.TextureMeta(atlas_offset=sum(len(a) for a in atlas), width=w, height=h, channels=3))
        coarse = rng.integers(lo, np.array(hi) + 1, size=(h // 8 + 1, w // 8 + 1, 3))
        atlas.append(np.repeat(np.repeat(coarse, 8, 0), 8, 1)[:h, :w].astype(np.uint8).reshape(-1))
    mats["diff_index"], mats["metal_rough_index"], mats["norm_index"] = 0, 1, 2
    atlas = np.concatenate(atlas)
    metas = (A.TextureMeta * len(metas))(*metas)
    sc = A.Scene.from_buffer_copy(scene.scene)
    sc.triangles = C.cast(tris.ctypes.data, C.POINTER(A.Triangle))
    sc.materials = C.cast(mats.ctypes.data, C.POINTER(A.Material))
    sc.tex_meta, sc.n_textures = metas, len(metas)
    sc.tex_atlas, sc.tex_atlas_bytes = C.cast(atlas.ctypes.data, C.POINTER(C.c_uint8)), atlas.size
    return P.SceneData(sc, keep=(scene, tris, mats, metas, atlas))


def _spot(scene):
    """The scene with a spot light added to its own lights."""
    lights = np.concatenate([scene.lights(), scene.lights()[:1]])
    verts = scene.triangle_vertices().reshape(-1, 3)
    lo, hi = verts.min(0), verts.max(0)
    at, down = lo + (hi - lo) * np.float32([0.3, 0.9, 0.6]), np.float32([0.1, -1.0, -0.1])
    down /= np.float32(np.linalg.norm(down))
    new = lights[-1]
    new["kind"] = A.PHX_LIGHT_SPOT
    for field, v in (("position", at), ("direction", down), ("power", np.float32([1.0, 0.9, 0.7]))):
        new[field]["x"], new[field]["y"], new[field]["z"], new[field]["w"] = *v, 0.0
    new["aux"]["x"], new["aux"]["y"], new["aux"]["z"], new["aux"]["w"] = 0.4, 0.7, 0.0, 0.0
    sc = A.Scene.from_buffer_copy(scene.scene)
    sc.lights, sc.n_lights = C.cast(lights.ctypes.data, C.POINTER(A.Light)), len(lights)
    sc.lum_pref_sum = None  # summed by the library over the new lights
    return P.SceneData(sc, keep=(scene, lights))


def _scene(case, seed):
    scene = P.SceneData.generate(KINDS[case["scene"]], seed=seed, width=case["width"], height=case["height"],
                                 detail=case["detail"])
    if case.get("maps"):
        scene = _maps(scene, seed)
    if case.get("spot"):
        scene = _spot(scene)
    return scene


def _args(case, seed):
    kind = case["scene"]
    return P.ArgsList(width=case["width"], height=case["height"], photons_per_round=case["photons"],
                      max_photon_bounces=DEPTH[kind], grid_res=GRID[kind], seed=seed & 0x7FFFFFFF,
                      direct_samples=case["samples"])


def _batch_members(case):
    """Uneven scenes of the three kinds: sides of half to the whole side, a quarter of the photons up;
    `mix` fixes which sizes they get."""
    rng = np.random.default_rng(case["mix"])
    for i in range(case["scenes"]):
        kind = list(KINDS)[i % 3]
        side = int(rng.integers(case["side"] // 2, case["side"] + 1))
        yield {"scene": kind, "detail": {"cornell": 0, "caustic": int(rng.choice([16, 32, 64])),
                                         "atrium": int(rng.choice([4, 8]))}[kind],
               "width": side, "height": side, "photons": int(rng.integers(case["photons"] // 4, case["photons"] + 1)),
               "samples": 16}


def prepare(case, seed):
    if case["op"] == "denoise":
        # a rendered image's noise: smooth shading, grain, a few fireflies
        rng = np.random.default_rng(seed)
        h, w = case["height"], case["width"]
        base = rng.integers(30, 200, size=(h // 40 + 1, w // 40 + 1, 3))
        img = np.repeat(np.repeat(base, 40, 0), 40, 1)[:h, :w] + rng.integers(-25, 26, size=(h, w, 3))
        img[rng.random((h, w)) < 0.002] = 255
        return {"case": case, "img": np.clip(img, 0, 255).astype(np.uint8)}
    if case["op"] == "batch":
        members = [(c, seed + 1 + i) for i, c in enumerate(_batch_members(case))]
        return {"case": case, "batch": P.Batch([_scene(c, s) for c, s in members], [_args(c, s) for c, s in members])}
    scene = _scene(case, seed)
    r = P.Renderer(_args(case, seed))
    r.set_scene(scene)
    if case["op"] == "render":
        return {"case": case, "r": r, "seeds": np.random.default_rng(seed)}
    # the optimiser's state: a start away from the truth, and the target rendered at the truth
    table = ParamTable(scene.materials(), scene.lights())
    rng0 = r.read("ROUND_RNG")
    target = torch.from_numpy(r.adjoint_forward(case["rounds"]))
    theta = table.vector()
    theta[:4 * table.n_mat] = 0.5 * theta[:4 * table.n_mat] + 0.25
    theta[4 * table.n_mat:] *= 0.8
    table.apply(r, theta)
    return {"case": case, "r": r, "table": table, "rng0": rng0, "target": target,
            "theta": torch.from_numpy(theta).requires_grad_(True)}


def run(state):
    case = state["case"]
    if case["op"] == "denoise":
        if case["filter"] == "mean":
            return denoise.mean_filter_gpu(state["img"], k=case["k"])
        if case["filter"] == "median":
            return denoise.median_filter_gpu(state["img"], k=case["k"])
        return denoise.gaussian_filter_gpu(state["img"], k=case["k"], sd=case["sd"])
    if case["op"] == "batch":
        b = state["batch"]
        b.iterate(case["rounds"])
        return [b.image(s) for s in range(b.n)]
    r = state["r"]
    if case["op"] == "render":
        if case["form"] == "seeded":
            for _ in range(case["rounds"]):
                r.round_seeded(int(state["seeds"].integers(0, 1 << 32)))
                shown = r.image_u8()
            return shown
        if case["form"] == "passes":
            for _ in range(case["rounds"]):
                r.round()
        else:
            r.iterate(case["rounds"])
        return r.image()
    # every step renders with the same round seeds
    r.write("ROUND_RNG", state["rng0"])
    theta = state["theta"]
    theta.grad = None
    img = render(theta, r, state["table"], case["rounds"])
    loss = ((img - state["target"]) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach(), "image": img.detach(), "grad": theta.grad}


def _triangles(case):
    d = case["detail"]
    if case["scene"] == "cornell":
        return 12
    if case["scene"] == "caustic":
        side = d or 256
        return 2 * (side - 1) ** 2 + 2 * max(6, side * 100 // 256) ** 2 + 12
    seg = d or 64
    return 17100 + 96 * seg * max(8, seg * 40 // 64)


def _round_work(case):
    """Bytes and operations of one round of one scene.  Bytes: the triangles, the SPPM state read and
    written (36 B a pixel), each stored photon written and read once (24 B).  Operations: one descent
    of a tree over the triangles (two box tests of 18 a level) and one triangle test (40) for each
    camera ray, each direct-lighting sample and each photon segment (about three a path)."""
    px, tris = case["width"] * case["height"], _triangles(case)
    stored = STORED[case["scene"]] * case["photons"]
    rays = px * (1 + case["samples"]) + 3 * case["photons"]
    return {"bytes": 108 * tris + 72 * px + 48 * stored, "flops": rays * (36 * math.log2(tris) + 40)}


def work(case):
    if case["op"] == "denoise":
        px, taps = case["width"] * case["height"], (2 * case["k"] + 1) ** 2
        return {"bytes": px * 3 * (1 + 8), "flops": px * 3 * taps}
    if case["op"] == "batch":
        rounds = [_round_work(c) for c in _batch_members(case)]
        return {k: case["rounds"] * sum(w[k] for w in rounds) for k in ("bytes", "flops")}
    w = _round_work(case)
    # the image leaves as 12 bytes a pixel (3 as shown); a backward pass replays the paths once more
    # and takes the image's gradient in
    out = case["width"] * case["height"] * (3 if case.get("form") == "seeded" else 12)
    passes = 2 if case["op"] == "inverse" else 1
    return {"bytes": passes * (case["rounds"] * w["bytes"] + out), "flops": passes * case["rounds"] * w["flops"]}


def exact(case, seed):
    """The filters in 64 bits.  A render is a random walk whose branches follow the rounding of each
    step, so no 64-bit value of it exists; its outputs are compared as they are."""
    if case["op"] != "denoise":
        return None
    a = prepare(case, seed)["img"].astype(np.float64)
    h, w, _ = a.shape
    k = case["k"]
    pad = np.full((h + 2 * k, w + 2 * k, 3), np.nan)
    pad[k:h + k, k:w + k] = a
    win = [pad[k + dy:h + k + dy, k + dx:w + k + dx] for dy in range(-k, k + 1) for dx in range(-k, k + 1)]
    if case["filter"] == "mean":
        return np.nanmean(np.stack(win), axis=0)
    if case["filter"] == "median":
        out = np.empty_like(a)
        for y in range(0, h, 64):  # a few rows at a time; the values outside the image sort last
            rows = np.sort(np.stack([v[y:y + 64] for v in win]), axis=0)
            n = np.sum(~np.isnan(rows), axis=0, keepdims=True)
            out[y:y + 64] = 0.5 * (np.take_along_axis(rows, (n - 1) // 2, 0) + np.take_along_axis(rows, n // 2, 0))[0]
        return out
    g = np.array([[math.exp(-(dx * dx + dy * dy) / (2.0 * case["sd"] ** 2)) for dx in range(-k, k + 1)]
                  for dy in range(-k, k + 1)])
    g /= g.sum()
    return sum(np.nan_to_num(v) * wt for v, wt in zip(win, g.reshape(-1)))
