"""Rays with a zero x component visit a box around their x without a look at y and z only
where some triangle's lower x face lies exactly at that x (where the reference's slab test
meets a NaN and accepts); elsewhere y and z prune.  Origins on lower and upper faces, between
faces, at both zeros and beside a non-finite triangle must all get the exhaustive search's
records."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS


def _scene(kind):
    tris = W.soup_tris(41, 9_000).reshape(-1, 3, 3)
    if kind == "grid":  # faces shared by many triangles, flat boxes, x = 0 among them
        tris = (np.round(tris * 16.0) / 16.0).astype(np.float32)
        tris[::2, :, 0] = tris[::2, :1, 0]
        tris[5, :, 0] = -0.0
    if kind == "nonfinite":
        tris[123, 1, 2] = np.inf
        tris[4567, 0, 0] = np.nan
    return np.ascontiguousarray(tris.reshape(-1, 9), dtype=np.float32)


def _rays(tris, n):
    rays = W.soup_rays(42, n).copy()
    x = tris.reshape(-1, 3, 3)[:, :, 0]
    k = np.arange(n) % len(x)
    rays[:, 3] = np.where(np.arange(n) % 3 == 0, -0.0, 0.0)
    rays[5::17, 3] = 1e-40  # (reciprocal infinite as well)
    rays[0::7, 0] = x.min(1)[k][0::7]
    rays[1::7, 0] = x.max(1)[k][1::7]
    rays[2::7, 0] = 0.0
    rays[3::7, 0] = -0.0
    rays[4::7, 0] = np.nextafter(x.min(1)[k][4::7], np.float32(-np.inf))
    rays[::11, 4] = 0.0
    rays[3::13, 3] = 0.1
    return rays


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 1)])
@pytest.mark.parametrize("kind", ["soup", "grid", "nonfinite"])
def test_zero_x_component(gpu_backend, oracle_lib, kind, leaf, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    tris = _scene(kind)
    rays = _rays(tris, 3_000)
    want = oracle_lib.brute_force(tris, rays)
    v = want["valid"] != 0
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(tris)
        b.set_option("node_format", fmt)
        for reps in (1, 750):  # one launch, two passes
            d = torch.from_numpy(np.tile(rays, (reps, 1))).cuda()
            rec = torch.zeros(len(d) * lay.size, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            b.nearest_hits_dev(d.data_ptr(), len(d), rec.data_ptr(), TAGS)
            b.sync()
            rec = rec.reshape(reps, -1)
            assert bool((rec == rec[0]).all())
            got = rec[0].cpu().numpy().view(lay.numpy_dtype())
            assert np.array_equal(got["valid"], want["valid"])
            assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
            assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)


def test_faces_follow_the_scene(gpu_backend, oracle_lib):
    """A smaller and a larger scene after one another: each build's own faces count."""
    for seed, n in ((51, 20_000), (52, 5_000), (53, 300), (54, 30_000)):
        tris = W.soup_tris(seed, n)
        rays = W.soup_rays(seed, 500).copy()
        rays[:, 3] = 0.0
        rays[::2, 0] = tris.reshape(-1, 3, 3)[:, :, 0].min(1)[:len(rays[::2])]
        gpu_backend.set_tris(tris)
        got, want = gpu_backend.nearest_hits(rays, TAGS), oracle_lib.brute_force(tris, rays)
        assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
        assert np.array_equal(got["valid"], want["valid"])
