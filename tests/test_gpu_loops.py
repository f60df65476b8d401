"""The two bounce loops (on the device without callbacks, window by window with
them) and the graphs that a scene keeps between calls."""
import pytest

from atrc_b200 import Config, DeviceScene, Film

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
