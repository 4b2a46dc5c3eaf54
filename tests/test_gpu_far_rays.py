"""Rays from far away (up to a million times the scene's extent), whose batches take the box test
without a margin past a distance that the build keeps for each scene: the exhaustive search's
records in every kind of build, beside ordinary rays, from buffers and in a batch of scenes."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W
from portablert_gb300._lib import Query
from portablert_gb300.batch import Batch, make_query

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS
M = 3000


def _rays(tris, seed):
    r = np.random.default_rng(seed)
    v = tris.reshape(-1, 3, 3).astype(np.float64)
    k = r.integers(0, len(v), M)
    w = r.dirichlet([1, 1, 1], M)
    target = (v[k] * w[:, :, None]).sum(1)
    d = r.normal(size=(M, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    away = 10.0 ** (np.arange(M) // 32 % 8 - 1.0)  # whole batches of a distance
    away[M // 2:] = 10.0 ** r.uniform(-1, 6, M - M // 2)
    o = target - d * away[:, None] * np.ptp(v.reshape(-1, 3), axis=0).max()
    d[::17, 1] = 0.0
    return np.concatenate([o, d], 1).astype(np.float32)


def _same(got, want):
    v = want["valid"] != 0
    assert np.array_equal(got["valid"], want["valid"])
    assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
    assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])
    for f in ("u", "v", "px", "py", "pz"):
        assert np.array_equal(got[f][v].view(np.uint32), want[f][v].view(np.uint32)), f


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (1, 1)])
@pytest.mark.parametrize("n,sah", [(1, 1), (2, 1), (3000, 1), (3000, 0), (9000, 1), (9000, 0)])
def test_far_rays(gpu_backend, oracle_lib, n, sah, leaf, fmt):
    b = gpu_backend
    tris = W.soup_tris(111, n) + np.float32(3.0)
    rays = _rays(tris, 112)
    want = oracle_lib.brute_force(tris, rays)
    assert np.count_nonzero(want["valid"]) > M // 8
    try:
        b.set_option("build_sah", sah)
        b.set_option("leaf_size", leaf)
        b.set_tris(tris)
        b.set_option("node_format", fmt)
        _same(b.nearest_hits(rays, TAGS), want)
    finally:
        b.set_option("build_sah", 1)
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)


@pytest.mark.parametrize("graph", [False, True])
def test_batch_of_scenes(gpu_backend, oracle_lib, graph):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    scenes = [W.soup_tris(120 + k, n) * np.float32(s) for k, (n, s) in
              enumerate([(500, 1.0), (1, 1.0), (7000, 1e-3), (60, 1e5)])]
    rays = [_rays(t, 130 + k) for k, t in enumerate(scenes)]
    off = np.concatenate([[0], np.cumsum([len(t) for t in scenes])]).astype(np.uint64)
    d_tris = torch.from_numpy(np.ascontiguousarray(np.concatenate(scenes), np.float32)).cuda()
    d_rays = torch.from_numpy(np.concatenate(rays)).cuda()
    rec = torch.zeros(len(d_rays) * lay.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    qs = (Query * len(scenes))(*[make_query(k, d_rays.data_ptr() + 24 * M * k, M,
                                            rec.data_ptr() + lay.size * M * k, TAGS)
                                 for k in range(len(scenes))])
    batch = Batch(b)
    try:
        if graph:
            batch.run_graph(d_tris.data_ptr(), off, qs)
        else:
            batch.set_tris_dev(d_tris.data_ptr(), off)
            batch.query_dev(qs)
        batch.sync()
    finally:
        batch.close()
    got = rec.cpu().numpy().view(lay.numpy_dtype())
    for k, t in enumerate(scenes):
        _same(got[k * M:(k + 1) * M], oracle_lib.brute_force(np.ascontiguousarray(t, np.float32), rays[k]))
