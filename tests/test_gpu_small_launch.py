"""Queries of few rays run as one launch whose batches of 4 or 8 rays are dealt out by warp,
each with the plain or the general box test; larger ones as a regular and a deferred pass.
The same rays, zero direction components among them, must get the same records either way,
at the sizes where batch, warp count and route change."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu

BIG = 400_000


def _rays():
    r = W.soup_rays(7, 20_000)
    r[5::97, 3] = 0.0
    r[11::301, 4:6] = 0.0
    r[4000:4032, 5] = 0.0
    r[777, 0] = np.nan
    return np.ascontiguousarray(np.concatenate([r] * (BIG // len(r))))


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (1, 1), (8, 1)])
@pytest.mark.parametrize("tags", [hitreg.TAGS, ("t",), ("valid",)])
def test_small_equals_large(gpu_backend, oracle_lib, leaf, fmt, tags):
    import torch

    b, lay = gpu_backend, hitreg.layout(tags)
    tris = W.soup_tris(8, 6000)
    rays = _rays()
    d = torch.from_numpy(rays).cuda()
    want = torch.zeros(BIG * lay.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    warps = int(b.stat("sms")) * 32
    sizes = [1, 2, 3, 4, 5, 7, 8, 9, 31, 33, 1000, 4 * warps - 1, 4 * warps, 4 * warps + 1,
             8 * warps + 3, 32 * warps, 32 * warps + 1, 200_001]
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(tris)
        b.set_option("node_format", fmt)
        b.nearest_hits_dev(d.data_ptr(), BIG, want.data_ptr(), tags)
        b.sync()
        for n in sizes:
            for off in (0, 4):
                got = torch.full(((n + 1) * lay.size + off,), 7, dtype=torch.uint8, device="cuda")
                torch.cuda.synchronize()
                b.nearest_hits_dev(d.data_ptr(), n, got.data_ptr() + off, tags)
                b.sync()
                assert torch.equal(got[off:off + n * lay.size], want[:n * lay.size]), (n, off)
                assert bool((got[off + n * lay.size:] == 7).all()) and bool((got[:off] == 7).all())
        if tags == hitreg.TAGS and fmt == 0:
            full = oracle_lib.brute_force(tris, rays[:2000])
            rec = want[:2000 * lay.size].cpu().numpy().view(lay.numpy_dtype())
            assert np.array_equal(rec["t"].view(np.uint32), full["t"].view(np.uint32))
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)
