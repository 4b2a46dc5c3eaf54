"""A query runs as one kernel with batches of 4, 8, 16 or 32 rays, the later ones claimed from a
counter, or as a regular and a deferred pass; a camera as one kernel without or with packet
descents.  The same rays must get the same records at the sizes where batch and route change."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W
from portablert_gb300._lib import Camera

pytestmark = pytest.mark.gpu

TAGS = ("t", "primitive_id", "valid")
TILE = 20_000


def _rays():
    r = W.soup_rays(61, TILE)
    r[5::997, 3] = 0.0
    r[11::3001, 4:6] = 0.0
    r[777, 0] = np.nan
    return np.ascontiguousarray(r)


@pytest.mark.parametrize("leaf,fmt,n_tris", [(1, 0, 5000), (1, 0, 700), (4, 0, 5000),
                                             (1, 1, 5000), (8, 1, 5000), (8, 1, 700)])
def test_routes_give_the_same_records(gpu_backend, oracle_lib, leaf, fmt, n_tris):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    tris, rays = W.soup_tris(62, n_tris), _rays()
    full = oracle_lib.brute_force(tris, rays[:1500])
    warps = int(b.stat("sms")) * 32
    sizes = [8 * warps, 8 * warps + 1, 16 * warps, 16 * warps + 5, 64 * warps, 64 * warps + 1,
             130 * warps - 3, 130 * warps + 1, 300 * warps, 300 * warps + 1, 420 * warps,
             420 * warps + 1]
    top = 421 * warps
    d = torch.from_numpy(np.tile(rays, (-(-top // TILE), 1))[:top]).cuda()
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(tris)
        b.set_option("node_format", fmt)
        want = torch.zeros(TILE, lay.size, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        b.nearest_hits_dev(d.data_ptr(), TILE, want.data_ptr(), TAGS)
        b.sync()
        rec = want[:1500].cpu().numpy().reshape(-1).view(lay.numpy_dtype())
        assert np.array_equal(rec["t"].view(np.uint32), full["t"].view(np.uint32))
        for n in sizes:
            got = torch.full((n + 1, lay.size), 7, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            for _ in range(2):  # (the counter starts again)
                b.nearest_hits_dev(d.data_ptr(), n, got.data_ptr(), TAGS)
            b.sync()
            whole = n // TILE * TILE
            assert bool((got[:whole].view(-1, TILE, lay.size) == want).all()), n
            assert torch.equal(got[whole:n], want[:n - whole]), n
            assert bool((got[n] == 7).all())
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("n,w,h", [(1, 1024, 600), (9, 1023, 601), (900, 1025, 601),
                                   (4097, 2049, 1281), (30_000, 700, 500),
                                   (30_000, 1500, 1000), (5_000, 2048, 1100)])
def test_camera_routes(gpu_backend, n, w, h, fmt):
    import torch

    b, lay, m = gpu_backend, hitreg.layout(TAGS), w * h
    c = Camera()
    c.width, c.height, c.form = w, h, 0
    c.pos[:] = [0.0, 0.05, -3.0]
    c.sensor_size, c.sensor_dist, c.sensor_z = 2.0, 2.0, -1.0
    try:
        b.set_tris(W.soup_tris(63, n) * np.float32(0.5))
        b.set_option("node_format", fmt)
        rays = torch.empty(m * 6, dtype=torch.float32, device="cuda")
        got = torch.zeros(m * lay.size, dtype=torch.uint8, device="cuda")
        want = torch.zeros_like(got)
        torch.cuda.synchronize()
        b.camera_rays(c, rays.data_ptr())
        b.nearest_hits_camera(c, got.data_ptr(), TAGS)
        b.nearest_hits_dev(rays.data_ptr(), m, want.data_ptr(), TAGS)
        b.sync()
        assert torch.equal(got, want)
    finally:
        b.set_option("node_format", 0)
