"""Top-level boxes shrunk to the instances' vertices lose no hit: seeded rays
against the oracle, for trees of one leaf (no node to shrink), one node and
several levels."""
import json

import pytest

from atrc_b200 import Config, DeviceScene
from atrc_b200.scenes import instanced_disney
from tests.parity import classify_closest, seeded_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instances", [1, 2, 4, 5, 33])
@pytest.mark.parametrize("builder", ["sah", "ploc"])
def test_shrunk_instances_lose_no_hit(tmp_path, instances, builder):
    import oracle
    path = instanced_disney(tmp_path / "inst", seed=7 + instances, ico_level=3, hf_res=24, instances=instances)
    d = json.loads(path.read_text())
    d["scene"]["bvh_builder"] = builder
    cfg = Config.from_string(json.dumps(d), path.parent)
    dev, ora = DeviceScene(cfg), oracle.OracleScene(cfg.scene_desc(), 3e-4)
    rays = seeded_rays(200_000, [-24] * 3, [24] * 3, [0, -27, 5], seed=instances)
    c = classify_closest(rays, dev.trace_rays(rays, "closest", exact=True), ora.trace_rays(rays), ora)
    assert c["error"] == 0, c
