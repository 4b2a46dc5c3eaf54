"""The small tier of the SAH build (tasks of at most 32 triangles, one warp each): nodes of 3
to 10 triangles sweep three axes in one pass, larger ones axis by axis, pairs are written
after the splits.  Sizes at those boundaries, triangles with equal centres (every order a
tie), flat scenes and one with a non-finite vertex, against the exhaustive search."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def sah(gpu_backend):
    gpu_backend.set_option("build_small", 0)
    yield gpu_backend
    gpu_backend.set_option("build_small", 1)
    gpu_backend.set_option("leaf_size", 1)


def _scene(kind, n):
    t = W.soup_tris(700 + n, n)
    if kind == "equal":
        t[: 2 * n // 3] = t[0]
    elif kind == "flat":
        t[:, 2::3] = np.float32(0.25)
        t[:, 1::3] *= np.float32(0.01)
    elif kind == "nan":
        t[n // 2, 3] = np.nan
    return t


@pytest.mark.parametrize("kind", ["soup", "equal", "flat", "nan"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9, 10, 11, 12, 19, 20, 21, 30, 31, 32, 45, 300])
def test_small_tasks(sah, oracle_lib, n, kind):
    tris = _scene(kind, n)
    rays = W.soup_rays(800 + n, 2000)
    rays[:, 3:] = tris.reshape(-1, 3, 3).mean(1)[np.arange(2000) % n] - rays[:, :3]
    rays[~np.isfinite(rays).all(1), 3:] = (0.0, 0.0, 1.0)
    want = oracle_lib.brute_force(tris, rays)
    assert (want["valid"] != 0).sum() >= 500  # of two triangles one may be the NaN one
    for leaf in (1, 4):
        sah.set_option("leaf_size", leaf)
        sah.set_tris(tris)
        got = sah.nearest_hits(rays, hitreg.TAGS)
        assert np.array_equal(got["valid"], want["valid"])
        assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
        v = want["valid"] != 0
        assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])
