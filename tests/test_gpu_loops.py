"""The two bounce loops (on the device without callbacks, window by window with
them) and the graphs that a scene keeps between calls."""
import numpy as np
import pytest

from atrc_b200 import Config, DeviceScene, Film
from atrc_b200.guide import Guide
from tests import kat_scenes as K

pytestmark = pytest.mark.gpu


def _seen(percent):
    pass


@pytest.mark.parametrize("progress", [None, _seen])
def test_iterations_are_counted_once(cornell_path, progress):
    cfg = Config.from_file(cornell_path)
    desc, _ = cfg.rendering(0)
    desc.width, desc.height, desc.spp = 40, 24, 3
    st = DeviceScene(cfg).render(desc, Film(40, 24), progress=progress)
    assert st["iterations"] == st["extend_launches"] > 0


def _same(a: Film, b: Film, what: str) -> None:
    # the same paths: only the order of the occlusion rays' FP32 additions and
    # of the film's FP64 ones differs
    np.testing.assert_allclose(a.weight, b.weight, rtol=1e-12, err_msg=what)
    for name in ("value", "value_sq", "albedo", "normal", "denoise"):
        x, y = getattr(a, name), getattr(b, name)
        assert (x is None) == (y is None)
        if x is not None:
            np.testing.assert_allclose(x, y, rtol=2e-6, atol=1e-6, err_msg=f"{what}: {name}")


def _feature_config(tmp_path):
    # sky, media, several lights and material types
    return Config.from_string(K.dumps(K.feature_scene(tmp_path, renderer="pt_cuda", spp=6, width=33, height=19)), tmp_path)


def test_windowed_loop_completes_like_the_device_loop(tmp_path):
    cfg = _feature_config(tmp_path)
    desc, _ = cfg.rendering(0)
    dev = DeviceScene(cfg)
    for pool in (0, 1000):  # more than one window of iterations
        desc.path_pool = pool
        ref = Film(desc.width, desc.height, value_sq=True, gbuffer=True)
        sr = dev.render(desc, ref)
        for call in range(2):  # the second call finds the first one's graph
            seen = []
            got = Film(desc.width, desc.height, value_sq=True, gbuffer=True)
            st = dev.render(desc, got, should_stop=lambda: False, progress=seen.append)
            for k in ("samples", "rays_closest", "rays_shadow", "iterations"):
                assert st[k] == sr[k], k
            assert seen == sorted(seen) and all(0 <= p <= 100 for p in seen)
            assert pool == 0 or len(seen) > 1
            _same(got, ref, f"pool {pool}, call {call}")


def test_kept_graphs_follow_the_call(tmp_path):
    """Calls that may and may not reuse a scene's graph, each against a scene
    of its own."""
    cfg = _feature_config(tmp_path)
    kept = DeviceScene(cfg)
    guide = Guide.for_scene(kept, log2_table=12)

    def call(scene, g, changes, gbuffer, callback, guided, record):
        desc, _ = cfg.rendering(0)
        for k, v in changes.items():
            setattr(desc, k, v)
        film = Film(desc.width, desc.height, value_sq=True, gbuffer=gbuffer)
        if guided:
            scene.render_guided(g, desc, film, record=record)
        else:
            scene.render(desc, film, progress=_seen if callback else None)
        return film

    steps = [({}, False, False, False, False), ({}, False, True, False, False), ({}, True, False, False, False),
             ({}, False, False, False, False), ({"eps": 1e-3}, False, False, False, False),
             ({"eps": 1e-3}, False, True, False, False), ({"disney_fixed": 1}, False, False, False, False),
             ({}, False, False, True, False), ({}, False, False, False, False), ({}, True, False, True, False),
             ({}, False, False, True, True), ({}, False, False, True, False), ({"path_pool": 200}, True, False, False, False),
             ({"path_pool": 5000, "width": 64, "height": 48}, True, True, False, False),
             ({"path_pool": 200}, True, True, False, False), ({"max_depth": 2}, False, False, False, False),
             ({"sort_mode": 0}, False, False, False, False), ({"isect_mode": 2}, False, True, False, False),
             ({"seed": 9}, False, False, False, False), ({}, False, True, False, False), ({}, False, False, False, False)]
    for i, (changes, gbuffer, callback, guided, record) in enumerate(steps):
        got = call(kept, guide, changes, gbuffer, callback, guided, record)
        fresh = DeviceScene(cfg)
        own = Guide.for_scene(fresh, log2_table=12) if guided else None
        _same(got, call(fresh, own, changes, gbuffer, callback, guided, record), f"step {i}: {steps[i]}")


@pytest.mark.parametrize("height", [255, 256])
def test_default_sort_starts_at_its_size(tmp_path, height):
    cfg = _feature_config(tmp_path)
    desc, _ = cfg.rendering(0)
    desc.width, desc.height, desc.spp, desc.task_grid_size = 512, height, 4, 4096
    dev = DeviceScene(cfg)
    films, launches = {}, {}
    for mode in (-1, 0, 1):
        desc.sort_mode = mode
        films[mode] = Film(desc.width, desc.height)
        st = dev.render(desc, films[mode])
        launches[mode] = st["kernel_launches"]
        assert st["samples"] == 512 * height * 4
    assert launches[-1] == launches[1 if height == 256 else 0] and launches[0] < launches[1]
    _same(films[-1], films[0], "auto")
    dev.set_tuning(sort_mode=2)  # chosen by the caller: at every size
    desc.sort_mode = -1
    assert dev.render(desc, Film(desc.width, desc.height))["kernel_launches"] == launches[1]
