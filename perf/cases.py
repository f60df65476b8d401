"""Timed calls of the renderer, for measuring a change of the code.

Each case is one call (or one frame's calls) that a program built on this
package makes in earnest, through its public entry points, on the seeded
scenes of ``atrc_b200.scenes``.  ``listed()`` gives the fixed cases, ``draw``
further ones of the same ranges, ``prepare`` what the program has in hand
before the call, ``run`` the call, ``work`` what it cannot do without and
``exact`` the results in 64 bits where they have such a value (ray queries on
the Cornell box; a path-traced image is one sample of a random variable, and
a trained network depends on such images).

A program loads a scene once and renders many frames of it, so the scenes are
kept for the life of the process; the seed draws the camera's place, the random
streams, the rays and the guide's parameters.
"""
from __future__ import annotations

import json
import math
import os
import tempfile
from pathlib import Path

import numpy as np
import torch

from atrc_b200 import RAY_DTYPE, Config, DeviceScene, Film, scenes
from atrc_b200.guide import Guide

# Per scene: closest-hit and occlusion rays of one camera sample (AO: the
# primary ray only), unique triangles, and the film sizes used in earnest.
SCENE_FACTS = {
    "cornell": {"closest": 4.5, "shadow": 3.5, "tris": 34},
    "cornell_sss": {"closest": 4.5, "shadow": 3.5, "tris": 34},
    "instanced": {"closest": 1.3, "shadow": 0.2, "tris": 3_076_098},
    "media": {"closest": 4.0, "shadow": 3.0, "tris": 200_040},
    "room": {"closest": 8.0, "shadow": 7.0, "tris": 403_000},
}
# Arithmetic of one ray and of one shaded vertex, about: a ray meets a dozen
# four-wide nodes (4 boxes x 12 flops) and two triangles (40 flops) on its way
# to the hit; a vertex evaluates and samples one BSDF and one light.
RAY_FLOPS, VERTEX_FLOPS = 12 * 48 + 2 * 40, 600


def listed() -> list:
    return [
        # the smallest frame: an editor's preview of a simple scene, one
        # sample per pixel, read back to the host each time
        {"name": "preview", "kind": "render", "scene": "cornell", "width": 64, "height": 64, "spp": 1, "host": True,
         "filter": "box", "gbuffer": False, "watertight": False},
        # the Cornell box at its full configuration (256 x 256 x 64 spp)
        {"name": "cornell", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 64, "host": True,
         "filter": "box", "gbuffer": False, "watertight": False},
        # one step of the instanced Disney + IBL frame (3.08M triangles)
        {"name": "instanced", "kind": "render", "scene": "instanced", "width": 1920, "height": 1080, "spp": 16,
         "host": False, "filter": "box", "gbuffer": False, "watertight": False},
        # long indirect paths: the indoor room, with the denoiser's G-buffer
        {"name": "room", "kind": "render", "scene": "room", "width": 1280, "height": 720, "spp": 4, "host": False,
         "filter": "box", "gbuffer": True, "watertight": False},
        # participating media (delta and ratio tracking), odd film size
        {"name": "media", "kind": "render", "scene": "media", "width": 767, "height": 511, "spp": 8, "host": False,
         "filter": "box", "gbuffer": False, "watertight": False},
        # subsurface scattering, watertight intersection, reconstruction by
        # the wide Gaussian filter
        {"name": "subsurface", "kind": "render", "scene": "cornell_sss", "width": 509, "height": 387, "spp": 8,
         "host": False, "filter": "gaussian", "gbuffer": False, "watertight": True},
        # ambient occlusion of the instanced scene
        {"name": "ao", "kind": "ao", "scene": "instanced", "width": 1280, "height": 720, "spp": 4, "host": False,
         "filter": "box", "gbuffer": False, "watertight": False},
        # many small views of one scene in one call (thumbnails, probes)
        {"name": "views", "kind": "batch", "scene": "room", "views": 16, "width": 128, "height": 96, "spp": 4},
        # one pass of the room with the learned guide (sampling only)
        {"name": "guided", "kind": "guided", "scene": "room", "width": 1280, "height": 720, "spp": 1},
        # the gradient of one training batch of the guide, forward and backward
        {"name": "learn", "kind": "learn", "scene": "room", "records": 200_003},
        # a large batch of incoherent closest-hit queries held on the device
        {"name": "queries", "kind": "rays", "scene": "instanced", "count": 4_000_003, "any": False, "exact": True,
         "host": False},
        # a small batch of host queries (picking, probes of a simple scene)
        {"name": "picks", "kind": "rays", "scene": "cornell", "count": 10_007, "any": False, "exact": True,
         "host": True},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["render"] * 5 + ["ao", "batch", "guided", "learn", "rays", "rays"])
    if kind == "rays":
        scene = rng.choice(["instanced", "room", "cornell"])
        return {"kind": kind, "scene": scene, "count": _log(rng, 1_000, 4_000_000), "any": rng.random() < 0.5,
                "exact": rng.random() < 0.5, "host": rng.random() < 0.3}
    if kind == "learn":
        return {"kind": kind, "scene": "room", "records": _log(rng, 2_000, 250_000)}
    width = _log(rng, 48, 1280 if kind != "batch" else 200)
    height = max(32, min(720, int(width * rng.uniform(0.45, 1.1))))
    if kind == "guided":
        return {"kind": kind, "scene": "room", "width": width, "height": height, "spp": 1}
    if kind == "batch":
        return {"kind": kind, "scene": "room", "views": rng.randint(3, 24), "width": width, "height": height,
                "spp": rng.choice([1, 2, 4])}
    scene = "instanced" if kind == "ao" else rng.choice(["cornell", "cornell_sss", "instanced", "media", "room"])
    most = 1_500_000 if scene in ("media", "room") else 3_000_000
    spp = max(1, min(_log(rng, 1, 64), most // (width * height)))
    return {"kind": kind, "scene": scene, "width": width, "height": height, "spp": spp, "host": rng.random() < 0.4,
            "filter": rng.choice(["box", "box", "gaussian"]), "gbuffer": rng.random() < 0.3,
            "watertight": rng.random() < 0.25}


# ------------------------------------------------------------------ scenes
_loaded: dict = {}


def _scene_file(name: str) -> Path:
    root = Path(tempfile.gettempdir()) / f"atrc_perf_scenes_{os.getuid()}"
    make = {"cornell": lambda d: scenes.cornell_box(d, renderer="pt_cuda"),
            "cornell_sss": lambda d: scenes.cornell_box(d, renderer="pt_cuda", subsurface=True),
            "instanced": scenes.instanced_disney, "media": scenes.media_scene, "room": scenes.indoor_room}[name]
    path = root / name / "scene.json"
    return path if path.exists() else make(root / name)


def _scene(name: str) -> tuple:
    if name not in _loaded:
        cfg = Config.from_file(_scene_file(name))
        _loaded[name] = (cfg, DeviceScene(cfg))
    return _loaded[name]


def _view(cfg, case: dict, rng, spread: float):
    """The scene's own view with the case's film, from a place nearby."""
    d, _ = cfg.rendering(0)
    d.width, d.height, d.spp = case["width"], case["height"], case["spp"]
    d.seed = int(rng.integers(1, 2 ** 31))
    for k in range(3):
        d.camera.pos[k] += float(rng.uniform(-spread, spread))
        d.camera.dst[k] += float(rng.uniform(-spread, spread))
    if case.get("filter") == "gaussian":
        d.filter_type, d.filter_radius, d.filter_alpha = 1, 1.5, 2.0
    d.isect_mode = 2 if case.get("watertight") else 0
    if case["kind"] == "ao":
        d.renderer, d.ao_sample_count, d.ao_max_distance = 1, 5, 2.0
        for k in range(3):
            d.ao_low[k], d.ao_high[k], d.ao_background[k] = 0.0, 1.0, 0.5
    return d


def prepare(case: dict, seed: int) -> dict:
    cfg, scene = _scene(case["scene"])
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    spread = 0.1 if case["scene"].startswith("cornell") else 0.3
    s = {"kind": kind, "scene": scene}
    if kind == "rays":
        rays = _rays(case, rng)
        if case["host"]:
            s["rays"] = rays
        else:
            s["rays"] = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
            s["hits"] = torch.empty((len(rays), 4), dtype=torch.float32, device="cuda")
        s |= {"host": case["host"], "mode": "any" if case["any"] else "closest", "exact": case["exact"]}
        return s
    if kind == "batch":
        s["descs"] = [_view(cfg, {**case, "width": case["width"] + 5 * k % 9}, rng, 1.0) for k in range(case["views"])]
        s["films"] = [Film(d.width, d.height, device=True) for d in s["descs"]]
        return s
    if kind == "learn":
        # a table that the gradient can be read back from at each call
        s["guide"] = Guide.for_scene(scene, seed=int(rng.integers(1, 2 ** 31)), log2_table=14)
        s["records"] = _records(case["records"], rng)
        return s
    s["desc"] = _view(cfg, case, rng, spread)
    if kind == "guided":
        s["film"] = Film(case["width"], case["height"], device=True)
        # a guide whose parameters have the spread that training gives them
        g = Guide.for_scene(scene, seed=int(rng.integers(1, 2 ** 31)))
        w, _ = g.params()
        g.set_params(weights=1.5 * w, table=rng.random(g.info()["table_floats"], np.float32) - 0.5)
        s["guide"] = g
        return s
    s["film"] = Film(case["width"], case["height"], gbuffer=case["gbuffer"], device=not case["host"])
    return s


def _unit(n: int, rng) -> np.ndarray:
    v = rng.standard_normal((n, 3), np.float32)
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _records(n: int, rng) -> np.ndarray:
    """Training records as a recording pass stores them: vertices of the room
    and what their paths brought back, most of it little, some of it much."""
    r = np.zeros((n, 24), np.float32)
    r[:, 0:3] = rng.uniform([-9.9, -5.9, 0.1], [9.9, 5.9, 7.9], (n, 3))
    r[:, 3:6], r[:, 6:9], r[:, 10:13] = _unit(n, rng), _unit(n, rng), _unit(n, rng)
    r[:, 9] = rng.uniform(0.02, 0.6, n)
    r[:, 13] = rng.uniform(0.05, 2.0, n)
    r[:, 14:17] = rng.uniform(0.1, 1.0, (n, 3))
    r[:, 17] = rng.lognormal(-2.0, 1.5, n)
    return r


def _rays(case: dict, rng) -> np.ndarray:
    n = case["count"]
    r = np.zeros(n, RAY_DTYPE)
    d = rng.standard_normal((n, 3), np.float32)
    if case["scene"] == "cornell":  # from the open side into the box
        r["o"] = rng.uniform([-0.3, -0.3, 3.5], [0.3, 0.3, 4.0], (n, 3))
        d = rng.uniform([-1, -1, -1], [1, 1, 1], (n, 3)).astype(np.float32) - r["o"]
    elif case["scene"] == "room":
        r["o"] = rng.uniform([-9, -5, 0.5], [9, 5, 7.5], (n, 3))
    else:
        r["o"] = rng.uniform(-20, 20, (n, 3))
    r["d"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["t_max"] = np.inf if not case["any"] else rng.uniform(1, 20, n)
    return r


# -------------------------------------------------------------------- calls
def _image(film: Film):
    """The picture of a film: value / weight, as Film.image() gives it on the host."""
    if not film.device:
        return film.image()
    v = film.value.view(film.height, film.width, 3)
    return (v / film.weight.view(film.height, film.width, 1).clamp_min(1e-30)).float()


def _outputs(film: Film) -> dict:
    out = {"image": _image(film), "weight": film.weight}
    if film.albedo is not None:  # the denoiser's inputs, in its 32 bits
        w = film.weight.reshape(-1, 1)
        for name, a in (("albedo", film.albedo), ("normal", film.normal), ("denoise", film.denoise)):
            v = a.reshape(len(w), -1) / w
            out[name] = v.float() if film.device else v.astype(np.float32)
    return out


def run(state: dict):
    kind, scene = state["kind"], state["scene"]
    if kind == "rays":
        if state["host"]:
            h = scene.trace_rays(state["rays"], state["mode"], exact=state["exact"])
            return {"t": h["t"], "entity": h["entity"], "prim": h["prim"], "u": h["u"]}
        rays, hits = state["rays"], state["hits"]
        scene.trace_rays_device(rays.data_ptr(), len(rays), hits.data_ptr(), state["mode"], exact=state["exact"])
        ids = hits.view(torch.int32)
        return {"t": hits[:, 0], "entity": ids[:, 1], "prim": ids[:, 2], "u": hits[:, 3]}
    if kind == "batch":
        for f in state["films"]:
            f.clear()
        scene.render_batch(state["descs"], state["films"])
        return [_image(f) for f in state["films"]]
    if kind == "learn":
        weights, table, loss = state["guide"].gradients(state["records"])
        return {"weights": weights, "table": table, "loss": np.float32(loss)}
    film = state["film"]
    film.clear()
    if kind == "guided":
        scene.render_guided(state["guide"], state["desc"], film)
    else:
        scene.render(state["desc"], film)
    return _outputs(film)


# --------------------------------------------------------------------- work
def work(case: dict) -> dict:
    facts = SCENE_FACTS[case["scene"]]
    # a triangle's three vertices, read by traversal
    geometry = facts["tris"] * 36
    if case["kind"] == "rays":
        n = case["count"]
        return {"bytes": n * 48 + geometry, "flops": n * RAY_FLOPS}
    if case["kind"] == "learn":  # records in, gradients of the table and the weights out
        n = case["records"]
        return {"bytes": n * 96 + 4 * (16 * (1 << 14) * 2 + 18_432), "flops": n * 110_592}
    pixels = case["width"] * case["height"] * case.get("views", 1)
    samples = pixels * case["spp"]
    # the film's value and weight; with the G-buffer seven more values
    film = pixels * 8 * (11 if case.get("gbuffer") else 4)
    if case["kind"] == "ao":
        return {"bytes": film + geometry, "flops": samples * 6 * RAY_FLOPS}
    rays = facts["closest"] + facts["shadow"]
    flops = samples * (rays * RAY_FLOPS + facts["closest"] * VERTEX_FLOPS)
    if case["kind"] == "guided":  # the network, at up to five vertices of a path
        flops += samples * 5 * 36_864
    return {"bytes": film + geometry, "flops": flops}


# -------------------------------------------------------------------- exact
def _cornell_triangles() -> np.ndarray:
    """(T, 3, 3) corners in 64 bits, in the order of the scene's entities."""
    path = _scene_file("cornell")
    tris = []
    for e in json.loads(path.read_text())["scene"]["entities"]:
        g = e["geometry"]
        if g["type"] == "quad":
            a, b, c, d = (np.array(g[k], np.float64) for k in "ABCD")
            tris += [np.stack([a, b, c]), np.stack([a, c, d])]
            continue
        raw = np.fromfile(path.parent / Path(g["filename"]).name, np.float32, offset=8)
        p = raw.reshape(-1, 3, 8)[..., :3].astype(np.float64)
        for t in reversed(g["transform"]):  # the last of the list is applied first
            if t["type"] == "rotate_y":
                c, s = math.cos(math.radians(t["deg"])), math.sin(math.radians(t["deg"]))
                p = p @ np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]]).T
            else:
                p = p + np.array(t["offset"], np.float64)
        tris += list(p)
    return np.array(tris)


def exact(case: dict, seed: int):
    if case["kind"] != "rays" or case["scene"] != "cornell":
        return None
    r = _rays(case, np.random.default_rng(seed))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tris = torch.from_numpy(_cornell_triangles()).to(dev)
    o, d = (torch.from_numpy(r[k].astype(np.float64)).to(dev) for k in ("o", "d"))
    t_max = torch.from_numpy(r["t_max"].astype(np.float64)).to(dev)
    best = t_max.clone()
    u = torch.zeros_like(best)
    hit = torch.zeros_like(best, dtype=torch.bool)
    for a, b, c in tris:
        e1, e2 = b - a, c - a
        s1 = torch.linalg.cross(d, e2.expand_as(d))
        div = s1 @ e1
        oa = o - a
        alpha = (oa * s1).sum(1) / div
        s2 = torch.linalg.cross(oa, e1.expand_as(oa))
        beta = (d * s2).sum(1) / div
        t = (s2 @ e2) / div
        on = (alpha >= 0) & (beta >= 0) & (alpha + beta <= 1) & (t >= 0) & (t < best)
        best, u, hit = torch.where(on, t, best), torch.where(on, alpha, u), hit | on
    miss = torch.full_like(best, -1.0)
    if case["any"]:
        return {"t": torch.where(hit, torch.ones_like(best), miss), "entity": None, "prim": None,
                "u": torch.zeros_like(u)}
    return {"t": torch.where(hit, best, miss), "entity": None, "prim": None, "u": torch.where(hit, u, torch.zeros_like(u))}
