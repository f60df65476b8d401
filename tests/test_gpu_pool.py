"""Path pools of every awkward size: camera rays that meet nothing end inside
the traversal kernel and leave their slot to the next sample, so a render must
take every sample once whatever the pool holds."""
import math

import numpy as np
import pytest

from atrc_b200 import Config, DeviceScene, Film
from tests import kat_scenes as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pool", [1, 15, 33, 1000, 4096 + 17])
@pytest.mark.parametrize("sort_mode, queue_order, fetch", [(0, 0, 0), (1, 1, 0), (2, 0, 1)])
def test_every_sample_is_taken_once(tmp_path, pool, sort_mode, queue_order, fetch):
    # 33 x 19 pixels of a scene with sky, media and several lights
    cfg = Config.from_string(K.dumps(K.feature_scene(tmp_path, renderer="pt_cuda", spp=5, width=33, height=19)), tmp_path)
    desc, _ = cfg.rendering(0)
    dev = DeviceScene(cfg)
    ref = Film(desc.width, desc.height, value_sq=True, gbuffer=True)
    desc.sort_mode, desc.path_pool = 0, 1 << 16
    sr = dev.render(desc, ref)
    dev.set_tuning(queue_order=queue_order, extend_fetch=fetch)
    desc.sort_mode, desc.path_pool = sort_mode, pool
    got = Film(desc.width, desc.height, value_sq=True, gbuffer=True)
    st = dev.render(desc, got)
    for k in ("samples", "rays_closest", "rays_shadow"):
        assert st[k] == sr[k], k
    np.testing.assert_array_equal(got.weight, ref.weight)
    # the same paths: only the order of the shadow rays' FP32 additions differs
    for name in ("value", "value_sq", "albedo", "normal", "denoise"):
        np.testing.assert_allclose(getattr(got, name), getattr(ref, name), rtol=2e-6, atol=1e-6, err_msg=name)


@pytest.mark.parametrize("min_depth, max_depth", [(2, 8), (0, 8), (0, 0)])
def test_camera_rays_into_a_white_sky(min_depth, max_depth):
    # the camera turns its back on the scene: every path is one ray.  With
    # roulette from the first vertex a sample is 0 or 1 / cont_prob, of mean 1
    cfg = Config.from_string(K.dumps(K.furnace(width=31, height=17, spp=64, renderer="pt_cuda")), ".")
    desc, _ = cfg.rendering(0)
    for k in range(3):
        desc.camera.dst[k] = 2 * desc.camera.pos[k] - desc.camera.dst[k]
    desc.min_depth, desc.max_depth, desc.cont_prob = min_depth, max_depth, 0.5
    dev = DeviceScene(cfg)
    f = Film(desc.width, desc.height, gbuffer=True)
    st = dev.render(desc, f)
    n = 31 * 17 * 64
    assert st["samples"] == st["rays_closest"] == n and st["rays_shadow"] == 0
    mean = f.value.sum() / (3 * f.weight.sum())
    if max_depth == 0:
        assert mean == 0
    elif min_depth > 0:
        np.testing.assert_allclose(f.image(), 1.0, rtol=1e-6)
    else:
        assert abs(mean - 1) < 5 / math.sqrt(n)  # variance of a sample: 1
    np.testing.assert_allclose(f.denoise, f.weight, rtol=1e-12)
    assert not f.albedo.any() and not f.normal.any()
