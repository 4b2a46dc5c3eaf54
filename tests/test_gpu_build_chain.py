"""Builds whose kernels are scheduled while the one before still runs: scenes of very
different sizes built in turn on one backend, so that whatever a kernel read too early
would be another scene's, with both builders, against the exhaustive search."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu


def _scene(n):
    nz = max(1, int((n / 4) ** 0.5))
    t = W.heightfield_tris(seed=n, nx=-(-n // (2 * nz)), nz=nz)[:n]
    return np.ascontiguousarray(t * np.float32(1 + n % 7) + np.float32(n % 11), np.float32)


def _rays(tris, m):
    rng = np.random.default_rng(len(tris))
    p = tris.reshape(-1, 3, 3).mean(1)[rng.integers(len(tris), size=m)]
    o = rng.uniform(-5, 5, (m, 3))
    d = p - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("sah", [0, 1])
@pytest.mark.parametrize("sizes", [(2, 9000, 33, 70_001), (513, 1, 20_000, 512), (1025, 1024)])
def test_builds_in_turn(gpu_backend, oracle_lib, sizes, sah):
    scenes = [_scene(n) for n in sizes]
    rays = [_rays(t, 400) for t in scenes]
    want = [oracle_lib.brute_force(t, r) for t, r in zip(scenes, rays)]
    try:
        gpu_backend.set_option("build_small", 0)
        gpu_backend.set_option("build_sah", sah)
        for _ in range(3):
            for t, r, w in zip(scenes, rays, want):
                gpu_backend.set_tris(t)
                got = gpu_backend.nearest_hits(r, hitreg.TAGS)
                v = w["valid"] != 0
                assert np.array_equal(got["valid"] != 0, v)
                assert np.array_equal(got["t"].view(np.uint32), w["t"].view(np.uint32))
                assert np.array_equal(got["primitive_id"][v], w["primitive_id"][v])
    finally:
        gpu_backend.set_option("build_sah", 1)
        gpu_backend.set_option("build_small", 1)
