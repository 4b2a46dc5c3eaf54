"""The camera's sensor coordinates without double arithmetic: the rays' bits against the
oracle's double expression, for widths whose quotients are exact or not, and sensor sizes
from denormal products to overflowing ones (those take the double path)."""
import numpy as np
import pytest

from portablert_gb300._lib import Camera

pytestmark = pytest.mark.gpu

SIZES = [0.05, -3.3, 1.0, 0.0, 1e-30, 1e-38, 1e-42, 1e30, 1e38, 3.4028235e38]


@pytest.mark.parametrize("width,height", [(1, 1), (3, 7), (8, 4), (1000, 3), (1919, 5), (4096, 2),
                                          (65537, 1), (1, 99991), (1 << 20, 1)])
def test_rays_have_the_double_expressions_bits(gpu_backend, oracle_lib, width, height):
    import torch

    n = width * height
    out = torch.empty(n * 6, dtype=torch.float32, device="cuda")
    for k, size in enumerate(SIZES):
        size = float(np.float32(size))
        c = Camera()
        c.width, c.height, c.form = width, height, k % 2
        c.pos[:] = [0.0, 0.0, 0.0]
        c.sensor_size, c.sensor_dist, c.sensor_z = size, 0.05, 0.05
        c.cos_a, c.sin_a = 1.0, 0.0
        torch.cuda.synchronize()
        gpu_backend.camera_rays(c, out.data_ptr())
        gpu_backend.sync()
        got = out.cpu().numpy().reshape(n, 6)
        want = oracle_lib.camera_rays(width, height, k % 2, (0.0, 0.0, 0.0), size, 0.05, 0.05, 1.0,
                                      0.0)
        nan = np.isnan(want)
        assert np.array_equal(nan, np.isnan(got))
        assert np.array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan]), size
