"""The SAH build's chunk sizes (256, 512 and 1,024 triangles per partition block, by scene
size): sizes on both sides of each change, in mesh order and shuffled, the larger first so
that the smaller ones use scratch reserved for it, against the exhaustive search."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu


def _scene(n, shuffled):
    nz = int((n / 4) ** 0.5)
    t = W.heightfield_tris(seed=n, nx=-(-n // (2 * nz)), nz=nz)[:n]
    if shuffled:
        t = t[np.random.default_rng(n).permutation(n)]
    return np.ascontiguousarray(t, np.float32)


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("edge", [256 * 608, 512 * 608])
def test_sizes_around_the_changes(gpu_backend, oracle_lib, edge, shuffled):
    for n in (edge + 1, edge, edge - 255):
        tris = _scene(n, shuffled)
        rng = np.random.default_rng(n)
        p = tris.reshape(-1, 3, 3).mean(1)[rng.integers(n, size=300)]
        o = rng.uniform(-5, 5, (300, 3))
        d = p - o
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        rays = np.concatenate([o, d], 1).astype(np.float32)
        want = oracle_lib.brute_force(tris, rays)
        gpu_backend.set_tris(tris)
        assert gpu_backend.stat("build_sah") == 1.0
        got = gpu_backend.nearest_hits(rays, hitreg.TAGS)
        v = want["valid"] != 0
        assert v.any()
        assert np.array_equal(got["valid"] != 0, v)
        assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
        assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])
