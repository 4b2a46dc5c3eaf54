"""The large and mid tiers of the SAH build: chunks of 1,024 triangles partitioned and binned
together, ranges of 33 to 512 triangles split in one block.  Sizes at those boundaries for
triangles in mesh order (whole warps in one bin), shuffled (many bins), in two piles and with
half of them identical, and a batch of scenes around the tier boundary, against the
exhaustive search."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W
from portablert_gb300.batch import Batch, make_query

pytestmark = pytest.mark.gpu


def _scene(kind, n):
    nz = max(1, int((n / 4) ** 0.5))
    t = W.heightfield_tris(seed=n, nx=-(-n // (2 * nz)), nz=nz)[:n]
    if kind == "shuffled":
        t = t[np.random.default_rng(n).permutation(n)]
    elif kind == "piles":
        t = t * np.float32(0.01)
        t[n // 3:, 0::3] += np.float32(7.0)
    elif kind == "half_equal":
        t[n // 2:] = t[n // 2]
    return np.ascontiguousarray(t, np.float32)


def _rays(tris, m):
    rng = np.random.default_rng(len(tris))
    p = tris.reshape(-1, 3, 3).mean(1)[rng.integers(len(tris), size=m)]
    o = rng.uniform(-5, 5, (m, 3))
    d = p + rng.normal(0, 0.01, (m, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


def _same(got, want):
    v = want["valid"] != 0
    assert np.array_equal(got["valid"] != 0, v)
    assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
    assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])


@pytest.mark.parametrize("kind", ["mesh", "shuffled", "piles", "half_equal"])
@pytest.mark.parametrize("n", [33, 40, 65, 127, 128, 129, 400, 511, 512, 513, 700, 1023, 1024,
                               1025, 1536, 2047, 2049, 3072, 9999, 70_001])
def test_tier_sizes(gpu_backend, oracle_lib, n, kind):
    tris = _scene(kind, n)
    rays = _rays(tris, 2000 if n < 20_000 else 400)
    want = oracle_lib.brute_force(tris, rays)
    try:
        gpu_backend.set_option("build_small", 0)
        gpu_backend.set_tris(tris)
        assert gpu_backend.stat("build_sah") == 1.0
        _same(gpu_backend.nearest_hits(rays, hitreg.TAGS), want)
    finally:
        gpu_backend.set_option("build_small", 1)


def test_scenes_across_the_tiers(gpu_backend, oracle_lib):
    import torch

    sizes = [(37 * s) % 1400 for s in range(150)] + [5000, 1, 0, 20_000]
    tris = [_scene("mesh" if s % 2 else "shuffled", n) if n else np.zeros((0, 9), np.float32)
            for s, n in enumerate(sizes)]
    lay = hitreg.layout(("t", "primitive_id", "valid"))
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    d_t = torch.from_numpy(np.concatenate(tris)).cuda()
    rays = W.camera_rays(16, 8)
    d_r = torch.from_numpy(rays).cuda()
    out = torch.zeros((len(sizes), 128 * lay.size), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    batch = Batch(gpu_backend)
    try:
        batch.set_tris_dev(d_t.data_ptr(), off)
        assert batch.stat("build_sah") == 1.0
        batch.query_dev([make_query(s, d_r.data_ptr(), 128, out[s].data_ptr(), lay.tags)
                         for s in range(len(sizes))])
        batch.sync()
        got = out.cpu().numpy()
        for s, t in enumerate(tris):
            _same(got[s].view(lay.numpy_dtype()), oracle_lib.brute_force(t, rays))
    finally:
        batch.close()


@pytest.mark.parametrize("n,ratio", [(3000, 1.01), (12_000, 1.003), (40_000, 1.001)])
def test_more_levels_than_halving(gpu_backend, oracle_lib, n, ratio):
    """Triangles at geometric distances: every split cuts off a few percent, so the trees need
    many more large levels than are queued before the first look at the counters.  The scene
    built before it is another one, so nothing left over from it may show."""
    rng = np.random.default_rng(n)
    x = ratio ** np.arange(n)
    t = rng.uniform(-0.3, 0.3, (n, 3, 3)) * x[:, None, None]
    t[:, :, 0] += x[:, None]
    tris = t.reshape(n, 9).astype(np.float32)
    k = rng.integers(n, size=600)
    o = np.stack([x[k], rng.uniform(-2, 2, 600) * x[k], 3 * x[k]], 1)
    d = tris.reshape(-1, 3, 3).mean(1)[k] - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    want = oracle_lib.brute_force(tris, rays)
    assert (want["valid"] != 0).sum() > 300
    try:
        gpu_backend.set_option("build_small", 0)
        for first in (W.soup_tris(1, 2 * n), tris):
            gpu_backend.set_tris(first)
        for leaf in (1, 4):
            gpu_backend.set_option("leaf_size", leaf)
            gpu_backend.set_tris(tris)
            _same(gpu_backend.nearest_hits(rays, hitreg.TAGS), want)
    finally:
        gpu_backend.set_option("build_small", 1)
        gpu_backend.set_option("leaf_size", 1)
