"""A query captured in a CUDA graph keeps the scene's buffers; after set_tris has built another
scene of at most as many triangles into them, a replay must give the new scene's records, also
where the box test looks up the scene's lower x faces (rays with a zero x component)."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS
N, RAYS = 9000, 6000


def _scene(seed, n):
    """Coordinates on a grid: many triangles have an edge in their box's lower x face, on which
    the reference's slab test accepts rays that point away as well."""
    return ((np.round(W.soup_tris(seed, n) * 16.0) + (seed % 7) / 8.0) / 16.0).astype(np.float32)


def _rays(*scenes):
    """Origins on lower x faces of the scenes' triangles, directions without an x component."""
    r = W.soup_rays(92, RAYS).copy()
    x = np.concatenate([t.reshape(-1, 3, 3)[:, :, 0].min(1) for t in scenes])
    r[:, 0] = x[np.arange(RAYS) * 7 % len(x)]
    r[:, 3] = np.where(np.arange(RAYS) % 2, 0.0, -0.0)
    r[::5] = W.soup_rays(93, RAYS)[::5]
    return np.ascontiguousarray(r)


def test_replay_after_rebuilds(gpu_backend, oracle_lib):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    first = _scene(90, N)
    others = [("sah", _scene(91, 5000)), ("lbvh", _scene(94, N)),
              ("one block", _scene(95, 3000)), ("sah", _scene(96, 7000))]
    rays = _rays(first, *[t for _, t in others])
    d = torch.from_numpy(rays).cuda()
    rec = torch.zeros(RAYS * lay.size, dtype=torch.uint8, device="cuda")
    s = torch.cuda.Stream()

    def query():
        b.nearest_hits_dev(d.data_ptr(), RAYS, rec.data_ptr(), TAGS, s.cuda_stream)

    def check(tris, what):
        want = oracle_lib.brute_force(tris, rays)
        got = rec.cpu().numpy().view(lay.numpy_dtype())
        assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32)), what
        hit = want["valid"] != 0
        assert np.array_equal(got["primitive_id"][hit], want["primitive_id"][hit]), what

    try:
        b.set_tris(first)
        torch.cuda.synchronize()
        query()
        b.sync()
        check(first, "first")
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            query()
        for how, tris in others:
            query()  # (set_tris waits for the stream's last query outside a capture)
            b.sync()
            b.set_option("build_sah", 0 if how == "lbvh" else 1)
            b.set_tris(tris)
            rec.zero_()
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            b.sync()
            check(tris, how)
    finally:
        b.set_option("build_sah", 1)
