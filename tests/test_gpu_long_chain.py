"""The bottom-up pass over a chain whose gaps grow all the way in finite floats: subtrees reach
over many blocks, and rays at every part of the chain, its far end among them, must get the
exhaustive search's records."""
import numpy as np
import pytest

from portablert_gb300 import hitreg

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS


@pytest.mark.parametrize("leaf,sah", [(1, 1), (4, 1), (1, 0)])
def test_chain(gpu_backend, oracle_lib, leaf, sah):
    n = 5000
    r = np.random.default_rng(141)
    x = np.cumsum(1.005 ** np.arange(n))  # up to about 1.4e13
    size = 1.005 ** np.arange(n)[:, None, None]
    t = r.uniform(-0.4, 0.4, (n, 3, 3)) * size
    t[:, :, 0] += x[:, None]
    tris = t.reshape(n, 9).astype(np.float32)
    k = np.linspace(0, n - 1, 1500).astype(int)
    w = r.dirichlet([1, 1, 1], len(k))
    target = (t[k] * w[:, :, None]).sum(1)
    d = r.normal(size=(len(k), 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([target - d * size[k, :, 0] * 2.0, d], 1).astype(np.float32)
    assert np.isfinite(tris).all() and np.isfinite(rays).all()
    want = oracle_lib.brute_force(tris, rays)
    assert np.count_nonzero(want["valid"][-300:]) > 150  # the far end too
    b = gpu_backend
    try:
        b.set_option("leaf_size", leaf)
        b.set_option("build_sah", sah)
        b.set_tris(tris)
        for fmt in (0, 1):
            b.set_option("node_format", fmt)
            got = b.nearest_hits(rays, TAGS)
            v = want["valid"] != 0
            assert np.array_equal(got["valid"], want["valid"])
            assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
            assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("build_sah", 1)
        b.set_option("node_format", 0)
