"""One-kernel queries whose batches after a warp's first one are smaller (four rays) or hold
twelve: at the sizes where batch, claim and route change, every tile of a query of repeated
rays must get the records of the exhaustive search, whoever took its batch."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu

TILE = 1000


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (8, 1)])
@pytest.mark.parametrize("tags", [hitreg.TAGS, ("t", "valid"), ("valid",)])
@pytest.mark.parametrize("tris", [700, 6000])
def test_every_tile_equals_the_exhaustive_search(gpu_backend, oracle_lib, tris, leaf, fmt, tags):
    import torch

    b, lay = gpu_backend, hitreg.layout(tags)
    scene = W.soup_tris(51, tris)
    rays = W.soup_rays(52, TILE).copy()
    rays[3::101, 3] = 0.0
    rays[7::211, 4] = -0.0
    rays[500, 2] = np.inf
    full = oracle_lib.brute_force(scene, rays)
    want = np.zeros(TILE, lay.numpy_dtype())
    for f in want.dtype.names:
        want[f] = full[f]
    warps = int(b.stat("sms")) * 32  # resident warps of the one kernel
    sizes = [8 * warps + 1, 8 * warps + 4, 9 * warps + 2, 32 * warps // 3, 32 * warps // 3 + 1,
             36 * warps, 36 * warps + 1, 50 * warps + 7, 64 * warps, 64 * warps + 1]
    most = max(sizes) + TILE
    d = torch.from_numpy(np.ascontiguousarray(np.tile(rays, (most // TILE + 1, 1)))).cuda()
    try:
        b.set_option("leaf_size", leaf)
        b.set_tris(scene)
        b.set_option("node_format", fmt)
        for n in sizes:
            got = torch.full(((n + 1) * lay.size,), 7, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            b.nearest_hits_dev(d.data_ptr(), n, got.data_ptr(), tags)
            b.sync()
            g = got.cpu().numpy()
            assert (g[n * lay.size:] == 7).all()
            rec = g[:n * lay.size].view(lay.numpy_dtype())
            for at in range(0, n, TILE):
                tile = rec[at:at + TILE]
                w = want[:len(tile)]
                if "valid" in tags:
                    assert np.array_equal(tile["valid"], w["valid"]), (n, at)
                if "t" in tags:
                    assert np.array_equal(tile["t"].view(np.uint32), w["t"].view(np.uint32)), (n, at)
                if "primitive_id" in tags:
                    hit = w["valid"] != 0
                    assert np.array_equal(tile["primitive_id"][hit], w["primitive_id"][hit]), (n, at)
    finally:
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)
