"""Queries large enough for a regular and a deferred pass, and images large enough for packet
descents (sizes from routes.py, whose routes test_routes_cpu.py checks without a GPU): batches
mixed of regular and other rays, every batch left to the deferred pass, leaves of several
triangles in both node formats, and packets whose rays part early."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W
from portablert_gb300._lib import Camera
from routes import packet_image, two_pass_rays

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS
TILE = 4000  # (not a multiple of 32: the other rays fall on every place of a batch)


def _rays(kind):
    r = W.soup_rays(71, TILE).copy()
    if kind == "mixed":
        r[5::160, 3] = 0.0
        r[77::352, 4] = -0.0
        r[77::352, 1] = 0.0
        r[1234, 0] = np.nan
        r[2345, 5] = 1e-30
    if kind == "deferred":  # one in every batch of 32, whatever the tile's offset
        r[::16, 5] = 0.0
    return np.ascontiguousarray(r)


def _check(rec, want, at):
    v = want["valid"] != 0
    assert np.array_equal(rec["valid"], want["valid"]), at
    assert np.array_equal(rec["t"].view(np.uint32), want["t"].view(np.uint32)), at
    assert np.array_equal(rec["primitive_id"][v], want["primitive_id"][v]), at
    for f in ("u", "v", "px", "py", "pz"):
        a, b = rec[f][v], want[f][v]
        assert ((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))).all(), (f, at)


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (1, 1), (8, 1)])
@pytest.mark.parametrize("kind", ["regular", "mixed", "deferred"])
def test_two_passes_against_exhaustive_search(gpu_backend, oracle_lib, kind, leaf, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    tris, rays = W.soup_tris(72, 9000), _rays(kind)
    want = oracle_lib.brute_force(tris, rays)
    n = two_pass_rays(int(b.stat("sms")), fmt, leaf)
    d = torch.from_numpy(rays).cuda().repeat(n // TILE + 1, 1)
    got = torch.full(((n + 1) * lay.size,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(tris)
        b.set_option("node_format", fmt)
        b.nearest_hits_dev(d.data_ptr(), n, got.data_ptr(), TAGS)
        b.sync()
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)
    whole = n // TILE
    first = got[:TILE * lay.size]
    _check(first.cpu().numpy().view(lay.numpy_dtype()), want, "first tile")
    assert bool((got[:whole * TILE * lay.size].view(whole, -1) == first).all())
    rest = n - whole * TILE
    assert torch.equal(got[whole * TILE * lay.size:n * lay.size], first[:rest * lay.size])
    assert bool((got[n * lay.size:] == 7).all())


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (1, 1), (8, 1)])
def test_one_kernel_equals_two_passes(gpu_backend, leaf, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    n = two_pass_rays(int(b.stat("sms")), fmt, leaf)
    rays = torch.from_numpy(_rays("mixed")).cuda().repeat(n // TILE + 1, 1)
    want = torch.zeros(n * lay.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(W.soup_tris(73, 6000))
        b.set_option("node_format", fmt)
        b.nearest_hits_dev(rays.data_ptr(), n, want.data_ptr(), TAGS)
        for m in (1, 5, 33, 1000, 20_000, 40_000, 200_001, 600_000):
            got = torch.zeros(m * lay.size, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            b.nearest_hits_dev(rays.data_ptr(), m, got.data_ptr(), TAGS)
            b.sync()
            assert torch.equal(got, want[:m * lay.size]), m
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)


def _camera(width, height):
    c = Camera()
    c.width, c.height, c.form = width, height, 0
    c.pos[:] = [0.0, 0.05, -3.0]
    c.sensor_size, c.sensor_dist, c.sensor_z = 2.0, 2.0, -1.0
    return c


def _bars(n, width):
    """Tall bars of two pixels at five columns of a 32-pixel row, pairs of them in each of many
    slabs behind one another: few rays of a packet share a bar, and each meets one in every
    slab."""
    r = np.random.default_rng(74)
    k = np.arange(n)
    depth = 2.0 + 0.02 * (k // 10) + 0.004 * (k % 2) + r.uniform(0, 0.002, n)
    column = 485 + 7 * (k // 2 % 5) + r.uniform(0, 1, n)
    x = (column / width - 0.5) * depth
    pixel = depth / width
    t = np.zeros((n, 3, 3))
    t[:, :, 0] = x[:, None] + pixel[:, None] * [0.0, 2.0, 1.0]
    t[:, :, 1] = depth[:, None] * [-1.0, -1.0, 1.0]
    t[:, :, 2] = depth[:, None] - 3.0
    return t.reshape(n, 9).astype(np.float32)


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (8, 0), (1, 1), (4, 1), (8, 1)])
@pytest.mark.parametrize("scene", ["soup", "bars", "one"])
def test_packets_equal_ray_buffer(gpu_backend, scene, leaf, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    n = 1 if scene == "one" else 900
    w, h = packet_image(int(b.stat("sms")), n)
    tris = _bars(n, w) if scene == "bars" else W.soup_tris(75, n)
    if scene == "one":
        tris[0] = [-1, -1, 0, 1, -1, 0, 0, 1, 0]
    m, cam = w * h, _camera(w, h)
    rays = torch.empty(m * 6, dtype=torch.float32, device="cuda")
    got = torch.zeros(m * lay.size, dtype=torch.uint8, device="cuda")
    want = torch.zeros_like(got)
    torch.cuda.synchronize()
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(tris)
        b.set_option("node_format", fmt)
        b.camera_rays(cam, rays.data_ptr())
        b.nearest_hits_camera(cam, got.data_ptr(), TAGS)
        b.nearest_hits_dev(rays.data_ptr(), m, want.data_ptr(), TAGS)
        b.sync()
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)
    assert torch.equal(got, want)
    hits = want.cpu().numpy().view(lay.numpy_dtype())["valid"]
    # (The bars cover 5 columns of a pixel or two in 1021.)
    assert np.count_nonzero(hits) > m // (300 if scene == "bars" else 100)
