"""Camera queries descend from the root in packets (the 32 rays of a warp on one node) before
single rays take over: every record must equal the one that the same rays get from a ray
buffer, whose traversal has no packets.  The dense soup overflows the packets' lists (a
pixel's ray passes hundreds of nodes), the narrow images make batches of 8 and 16 rays and a
ragged last one, the even widths put zero direction components into some batches."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W
from portablert_gb300._lib import Camera

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS


def _camera(width, height):
    c = Camera()
    c.width, c.height, c.form = width, height, 0
    c.pos[:] = [0.0, 0.05, -3.0]
    c.sensor_size, c.sensor_dist, c.sensor_z = 2.0, 2.0, -1.0
    return c


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (1, 1), (4, 0), (8, 1)])
@pytest.mark.parametrize("n", [1, 9, 4097, 60_000])
def test_camera_equals_ray_buffer(gpu_backend, n, leaf, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(W.soup_tris(17, n))
        b.set_option("node_format", fmt)
        for w, h in ((1, 1), (7, 5), (31, 33), (64, 48), (1023, 401)):
            cam, m = _camera(w, h), w * h
            rays = torch.empty(m * 6, dtype=torch.float32, device="cuda")
            got = torch.zeros(m * lay.size, dtype=torch.uint8, device="cuda")
            want = torch.zeros_like(got)
            torch.cuda.synchronize()
            b.camera_rays(cam, rays.data_ptr())
            b.nearest_hits_camera(cam, got.data_ptr(), TAGS)
            b.nearest_hits_dev(rays.data_ptr(), m, want.data_ptr(), TAGS)
            b.sync()
            assert torch.equal(got, want), (w, h)
            if m > 1000 and n > 1000:
                hits = want.cpu().numpy().view(lay.numpy_dtype())["valid"]
                assert np.count_nonzero(hits) > m // 20
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)
