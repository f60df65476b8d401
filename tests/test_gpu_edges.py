"""Rays that graze a triangle's edge alpha + beta = 1: the fast triangle test
decides them by the last bit of a sum, and the form of that sum (both terms
rounded for ray queries, one product fused for a render's occlusion rays) is
part of the results."""
import json

import numpy as np
import pytest

from atrc_b200 import RAY_DTYPE, Config, DeviceScene, Film
from tests import kat_scenes as K

A, B, C = np.array([[-1.125, -0.75, 0.375], [1.25, -0.5, -0.625], [-0.25, 1.375, 0.5]])
F = np.float32


def _fma(a, b, c):  # the product is exact in 64 bits
    return F(a.astype(np.float64) * b + c)


def _cross(a, b):
    return [_fma(a[i], b[j], -F(a[j] * b[i])) for i, j in ((1, 2), (2, 0), (0, 1))]


def _dot(a, b):
    return _fma(a[2], b[2], _fma(a[0], b[0], F(a[1] * b[1])))


def _edge_rays(n: int):
    """Rays at the middle of the edge BC, and which of them meet the triangle:
    alpha + beta with both terms rounded, and with one product fused."""
    rng = np.random.default_rng(17)
    r = np.zeros(n, RAY_DTYPE)
    s = rng.uniform(0.2, 0.8, (n, 1))
    r["o"] = rng.uniform([-2, -2, 2], [2, 2, 4], (n, 3))
    d = s * B + (1 - s) * C - r["o"]
    r["d"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["t_max"] = np.inf
    o, d = r["o"].T, r["d"].T
    ba, ca, oa = F(B - A), F(C - A), F(o - F(A)[:, None])
    s1 = _cross(d, ca)
    inv = F(1) / _dot(s1, ba)
    da = _dot(oa, s1)
    alpha, s2 = F(da * inv), _cross(oa, ba)
    db = _dot(d, s2)
    beta = F(db * inv)
    assert (alpha > 0.1).all() and (beta > 0.1).all()
    return r, F(alpha + beta) <= 1, _fma(da, inv, beta) <= 1, _fma(db, inv, alpha) <= 1


def _triangle_scene():
    d = K.edge_scene()
    d["scene"]["entities"][0]["geometry"] = {"type": "quad", "A": list(A), "B": list(B), "C": list(C), "D": list(A),
                                             "transform": []}
    return d


def test_edge_rays_tell_the_forms_apart():
    _, rounded, fused_a, fused_b = _edge_rays(100_000)
    assert 0.2 < rounded.mean() < 0.95
    assert (rounded != fused_a).mean() > 0.01 and (rounded != fused_b).mean() > 0.01 and (fused_a != fused_b).mean() > 0.01


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["closest", "any"])
def test_queries_round_both_terms(mode):
    rays, rounded, _, _ = _edge_rays(100_000)
    dev = DeviceScene(Config.from_string(json.dumps(_triangle_scene()), "."))
    hit = dev.trace_rays(rays, mode, exact=False)["entity"] >= 0
    # the emulation rounds a fused sum twice: about one ray in 2^29 apart
    assert np.array_equal(hit, rounded), int((hit != rounded).sum())


# Pixels of the indoor room that hold a path whose occlusion ray grazes an
# edge: seed of the render, the camera's shifts, pixel and value.
GRAZED = [
    (95492385, [0.17321582687648246, -0.27253320256813029, -0.14273201784113537],
     [0.13322673053416834, -0.10232584223471086, 0.03856410505992347], (100, 480), [0.3044708, 0.06917141, 0.03102251]),
    (1624127525, [0.13134639226062056, 0.25985319817201585, 0.099861984066265563],
     [-0.10132368530940286, -0.23710513542880374, 0.19155235608372168], (25, 712), [0.04275153, 0.01390731, 0.1779755]),
    (139998475, [-0.019012819069458897, -0.095808115284785, -0.20613480923332167],
     [0.20474020185112701, -0.06370704826902121, -0.042469117350815322], (884, 715), [0, 0, 0]),
    (1776046495, [0.14033376194726305, -0.0061208692940744602, 0.11094405533010004],
     [0.028977641445168789, 0.019133845054543963, -0.24438396859551634], (823, 523), [0.05257732, 0.03923597, 0.008826545]),
    (1082894378, [-0.29981277889739782, -0.079182421805900821, -0.18415027177943932],
     [-0.17004092132230983, -0.29878427519141865, 0.29451730734552412], (232, 535), [3.58366e-05, 5.601079e-05, 0.0002555258]),
]


@pytest.mark.gpu
@pytest.mark.parametrize("seed, pos, dst, pixel, value", GRAZED)
def test_occlusion_rays_keep_their_edges(scene_dir, seed, pos, dst, pixel, value):
    from atrc_b200.scenes import indoor_room
    cfg = Config.from_file(indoor_room(scene_dir / "room_edges"))
    desc, _ = cfg.rendering(0)
    desc.spp, desc.seed = 4, seed
    for k in range(3):
        desc.camera.pos[k] += pos[k]
        desc.camera.dst[k] += dst[k]
    film = Film(desc.width, desc.height)
    DeviceScene(cfg).render(desc, film)
    # the sums of a path's FP32 terms; a flipped edge changes the whole value
    np.testing.assert_allclose(film.image()[pixel[1], pixel[0]], value, rtol=1e-4, atol=1e-6)
