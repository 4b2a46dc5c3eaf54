"""Rays out of the ranges that the plain box test takes: components under 2^-58 beside zeros and
ordinary ones, directions up to the largest floats, origins past 2^67, alone and mixed.  Every
record must be the exhaustive search's, in both node formats, as one kernel and as two passes."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W
from routes import two_pass_rays

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS
M = 4096


def _scene(kind):
    t = W.soup_tris(101, 6000)
    if kind == "grid":  # faces that many origins lie on
        t = (np.round(t * 16.0) / 16.0).astype(np.float32)
    if kind == "large":
        t = (t * np.float32(2.0 ** 40)).astype(np.float32)
    return t


def _rays(tris):
    r = np.random.default_rng(102)
    scale = np.abs(tris).max()
    rays = W.soup_rays(103, M).astype(np.float64)
    rays[:, :3] *= scale
    v = tris.reshape(-1, 3)[r.integers(0, 3 * len(tris), M)]
    group = np.arange(M) // 32 % 8  # whole batches of a kind
    axis = r.integers(0, 3, M)
    at = np.arange(M), axis
    near = group >= 1
    rays[near, :3] = np.where(r.random((near.sum(), 3)) < 0.5, v[near], rays[near, :3])
    tiny = np.isin(group, (1, 2, 6))
    rays[:, 3:][at] = np.where(tiny, rays[:, 3:][at] * 2.0 ** r.uniform(-120, -59, M), rays[:, 3:][at])
    other = np.arange(M), (axis + 1) % 3
    rays[:, 3:][other] = np.where(group == 2, 0.0, rays[:, 3:][other])
    rays[group == 3, 3:] *= 2.0 ** r.uniform(61, 120, ((group == 3).sum(), 1))
    far = np.isin(group, (4, 6))
    rays[far, :3] -= rays[far, 3:] * 2.0 ** r.uniform(66, 100, (far.sum(), 1))
    rays[group == 5, :3] = 2.0 ** r.uniform(60, 127, ((group == 5).sum(), 3))
    with np.errstate(over="ignore"):
        rays = rays.astype(np.float32)
    last = group == 7  # any of them in one batch
    rays[last] = rays[r.permutation(M)[:last.sum()]]
    return np.ascontiguousarray(rays)


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (1, 1)])
@pytest.mark.parametrize("kind", ["soup", "grid", "large"])
def test_odd_rays(gpu_backend, oracle_lib, kind, leaf, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    tris = _scene(kind)
    rays = _rays(tris)
    want = oracle_lib.brute_force(tris, rays)
    hit = want["valid"] != 0
    assert hit.sum() > M // 20
    usual = np.ascontiguousarray(W.soup_rays(104, M) * [[np.abs(tris).max()] * 3 + [1] * 3], np.float32)
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(tris)
        b.set_option("node_format", fmt)
        for n in (M, two_pass_rays(int(b.stat("sms")), fmt, leaf)):
            d = torch.from_numpy(rays).cuda()
            if n > M:
                more = torch.from_numpy(usual).cuda().repeat(n // M + 1, 1)
                d = torch.cat([more[:n - M - 13], d, more[:13]])
            at = 0 if n == M else n - M - 13
            rec = torch.zeros(n * lay.size, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            b.nearest_hits_dev(d.data_ptr(), n, rec.data_ptr(), TAGS)
            b.sync()
            got = rec[at * lay.size:(at + M) * lay.size].cpu().numpy().view(lay.numpy_dtype())
            assert np.array_equal(got["valid"], want["valid"]), n
            assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32)), n
            assert np.array_equal(got["primitive_id"][hit], want["primitive_id"][hit]), n
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)
