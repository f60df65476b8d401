"""Top-level boxes shrunk to the instances' vertices keep every hit that the
rounded world -> entity transform finds: instances modelled far from their
origin and rays from far away, aimed past the extreme vertices by as much as
that transform rounds.  A scene of one entity has no top-level box, so a ray
meets something in the scene of all entities if it does with one of them alone.
(Occlusion: closest hits also depend on the order of the visits, by the slack of
the boxes against the nearest hit.)  The rotations tilt every axis, so that the
boxes of the instances' corners, too, keep all these hits."""
import json

import numpy as np
import pytest

from atrc_b200 import RAY_DTYPE, Config, DeviceScene
from atrc_b200.scenes import _icosahedron, write_bm

pytestmark = pytest.mark.gpu


def _sphere(levels: int) -> np.ndarray:
    v, f = _icosahedron()
    t = v[f]
    for _ in range(levels):
        a, b, c = t[:, 0], t[:, 1], t[:, 2]
        ab, bc, ca = a + b, b + c, c + a
        t = np.concatenate([np.stack(x, 1) for x in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca))])
        t /= np.linalg.norm(t, axis=2, keepdims=True)
    return t


# about z, then x, then y
ANGLES = [("rotate_y", 50.0), ("rotate_x", 40.0), ("rotate_z", 30.0)]


def _rotation() -> np.ndarray:
    m = np.eye(3)
    for name, deg in ANGLES:
        c, s = np.cos(np.radians(deg)), np.sin(np.radians(deg))
        i, j = {"x": (1, 2), "y": (2, 0), "z": (0, 1)}[name[-1]]
        r = np.eye(3)
        r[i, i], r[i, j], r[j, i], r[j, j] = c, -s, s, c
        m = m @ r
    return m


def _case(tmp_path, tris: np.ndarray, centre):
    """The mesh modelled around `centre`, rotated, and moved to each place.
    Returns the entities, a maker of scenes and the triangles of the world."""
    centre = np.array(centre, np.float64)
    t32 = (tris + centre).astype(np.float32)
    write_bm(tmp_path / "mesh.bm", t32, np.zeros_like(t32) + [0, 0, 1], np.zeros(t32.shape[:2] + (2,)))
    m = _rotation()
    ents, world = [], []
    for at in PLACES:
        off = (np.array(at) - m @ centre).tolist()
        ents.append({"type": "geometric", "material": {"type": "ideal_black"},
                     "geometry": {"type": "transform_wrapper",
                                  "transform": [{"type": "translate", "offset": off}] + [{"type": k, "deg": a} for k, a in ANGLES],
                                  "internal": {"type": "reference", "name": ["meshes", "mesh"]}}})
        world.append(t32.astype(np.float64) @ m.T + off)
    mesh = {"type": "triangle_bvh", "filename": "${scene-directory}/mesh.bm", "transform": []}
    d = {"scene": {"type": "default", "meshes": {"mesh": mesh}},
         "rendering": {"camera": {"type": "thin_lens", "pos": [0, 0, 3], "dst": [0, 0, 0], "up": [0, 1, 0], "fov": 40},
                       "width": 4, "height": 4, "renderer": {"type": "pt_cuda", "spp": 1}, "reporter": {"type": "noout"}}}

    def scene(entities):
        d["scene"]["entities"] = entities
        return DeviceScene(Config.from_string(json.dumps(d), tmp_path))
    return ents, scene, np.concatenate(world)


def _rays(world: np.ndarray, distance: float, past: float, n: int) -> np.ndarray:
    """At points within `past` of the outermost vertices along an axis, seen
    across that axis from `distance` away."""
    rng = np.random.default_rng(5)
    r = np.zeros(n, RAY_DTYPE)
    a, sign = rng.integers(0, 3, n), rng.choice([-1.0, 1.0], n)
    pts = world.reshape(-1, 3)
    order = {(k, s): np.argsort(-s * pts[:, k])[:24] for k in range(3) for s in (-1.0, 1.0)}
    p = pts[[order[k, s][rng.integers(0, 24)] for k, s in zip(a, sign)]]
    p[np.arange(n), a] += sign * rng.uniform(-past, past, n)
    d = rng.standard_normal((n, 3))
    d[np.arange(n), a] *= 1e-3
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r["o"] = p - distance * d
    d = p - r["o"].astype(np.float64)
    r["d"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["t_max"] = np.inf
    return r


PLACES = [(-3.0, 0.5, 0.25), (0.0, 0.0, 0.0), (3.5, -1.0, 0.75)]


@pytest.mark.parametrize("centre, distance", [((0, 0, 0), 4.0), ((5e4, 5e4, 0), 4.0), ((-7e3, 2e4, 9e3), 4.0),
                                              ((0, 0, 0), 60.0), ((0, 0, 0), 3e3), ((0, 0, 0), 1e5), ((300, 0, -200), 2e4)])
@pytest.mark.parametrize("isect", [0, 1, 2])
def test_hits_past_extreme_vertices(tmp_path, centre, distance, isect):
    ents, scene, world = _case(tmp_path, _sphere(2), centre)
    # a few ulp of the coordinates that the transform passes through
    past = 2.0 ** -21 * (np.abs(centre).max() + distance)
    rays = _rays(world, distance, past, 100_000)
    alone = np.any([scene([e]).trace_rays(rays, "any", isect=isect)["entity"] >= 0 for e in ents], axis=0)
    assert 0.2 < alone.mean() < 0.98
    lost = (scene(ents).trace_rays(rays, "any", isect=isect)["entity"] >= 0) != alone
    assert lost.sum() == 0, (int(lost.sum()), rays[lost][:3])
