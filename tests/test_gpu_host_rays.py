"""Host ray batches around the sizes at which atrc_cuda_trace_rays changes its
route (pinned stage, kept device buffer, buffers of the call's own)."""
import numpy as np
import pytest

from atrc_b200 import Config, DeviceScene
from tests.parity import seeded_rays

pytestmark = pytest.mark.gpu

STAGE, KEEP = 1 << 17, 1 << 20


@pytest.mark.parametrize("mode", ["closest", "any"])
def test_host_batches_equal_device_queries(cornell_path, mode):
    import torch
    dev = DeviceScene(Config.from_file(cornell_path))
    rays = seeded_rays(KEEP + 33, [-1.2] * 3, [1.2] * 3, [0, 0, 3.8], seed=5)
    if mode == "any":
        rays["t_max"] = 1.5
    d_rays = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
    d_hits = torch.empty((len(rays), 4), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    dev.trace_rays_device(d_rays.data_ptr(), len(rays), d_hits.data_ptr(), mode)
    want = d_hits.cpu().numpy().view(np.uint32)
    # growing, shrinking and growing again
    for n in (1, 31, 33, 1024, 1025, STAGE, STAGE + 1, 5, KEEP, KEEP + 33, 700, STAGE):
        got = dev.trace_rays(rays[:n], mode)
        assert np.array_equal(got.view(np.uint32).reshape(-1, 4), want[:n]), n
