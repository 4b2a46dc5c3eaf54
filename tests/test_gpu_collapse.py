"""The collapse to 8-wide nodes takes 32 items per block, eight lanes each, and writes nodes,
compressed nodes and triangle records together.  Batches whose levels end inside a block,
with empty and one-triangle scenes among the others, for both collapses, several leaf
sizes and both node formats, against the exhaustive search of each scene alone."""
import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W
from portablert_gb300.batch import Batch, make_query

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 7, 8, 9, 0, 63, 64, 65, 100, 300, 1, 520, 3, 1000]
COUNTS = [1, 31, 32, 33, 70]


@pytest.mark.parametrize("cost", [1, 0])
@pytest.mark.parametrize("leaf", [1, 3, 8])
@pytest.mark.parametrize("count", COUNTS)
def test_levels_across_blocks(gpu_backend, oracle_lib, count, leaf, cost):
    import torch

    b = gpu_backend
    sizes = [SIZES[(5 * s + count) % len(SIZES)] for s in range(count)]
    tris = [W.soup_tris(40 + s, n) for s, n in enumerate(sizes)]
    rays = W.soup_rays(41, 512)
    want = [oracle_lib.brute_force(t, rays) for t in tris]
    lay = hitreg.layout(("t", "primitive_id", "valid"))
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    d_t = torch.from_numpy(np.concatenate(tris + [np.zeros((1, 9), np.float32)])).cuda()
    d_r = torch.from_numpy(rays).cuda()
    out = torch.zeros((count, 512 * lay.size), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    batch = Batch(b)
    try:
        b.set_option("leaf_size", leaf)
        b.set_option("collapse_cost", cost)
        for graph in (False, True):
            for fmt in (0, 1):
                b.set_option("node_format", fmt)
                out.zero_()
                torch.cuda.synchronize()
                qs = [make_query(s, d_r.data_ptr(), 512, out[s].data_ptr(), lay.tags)
                      for s in range(count)]
                if graph:
                    batch.run_graph(d_t.data_ptr(), off, qs)
                else:
                    batch.set_tris_dev(d_t.data_ptr(), off)
                    batch.query_dev(qs)
                batch.sync()
                got = out.cpu().numpy()
                for s in range(count):
                    g = got[s].view(lay.numpy_dtype())
                    v = want[s]["valid"] != 0
                    assert np.array_equal(g["valid"] != 0, v), (s, graph, fmt)
                    assert np.array_equal(g["t"].view(np.uint32), want[s]["t"].view(np.uint32))
                    assert np.array_equal(g["primitive_id"][v], want[s]["primitive_id"][v])
    finally:
        batch.close()
        b.set_option("leaf_size", 1)
        b.set_option("collapse_cost", 1)
        b.set_option("node_format", 0)


@pytest.mark.parametrize("n", [2, 3, 255, 256, 257, 258, 511, 512, 513, 769, 5000])
@pytest.mark.parametrize("sah,cost", [(0, 0), (0, 1), (1, 1)])
def test_bottom_up_across_blocks(gpu_backend, oracle_lib, n, sah, cost):
    """The bottom-up pass finishes the nodes of 256 leaves in one block and walks the rest:
    scenes at the block boundary, one of them a chain of ever larger gaps (one deep tree)."""
    b = gpu_backend
    chain = W.soup_tris(60, n)
    chain[:, 0::3] = (chain[:, 0::3] + (1.02 ** np.arange(n))[:, None]).astype(np.float32)
    rays = W.soup_rays(61, 1000)
    rays_c = rays.copy()
    rays_c[:, 3:] = chain.reshape(-1, 3, 3).mean(1)[np.arange(1000) % n] - rays[:, :3]
    try:
        b.set_option("build_small", 0)
        b.set_option("build_sah", sah)
        b.set_option("collapse_cost", cost)
        for tris, r in ((W.soup_tris(62, n), rays), (chain, rays_c)):
            want = oracle_lib.brute_force(tris, r)
            b.set_tris(tris)
            got = b.nearest_hits(r, hitreg.TAGS)
            v = want["valid"] != 0
            assert np.array_equal(got["valid"], want["valid"])
            assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
            assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])
    finally:
        b.set_option("build_small", 1)
        b.set_option("build_sah", 1)
        b.set_option("collapse_cost", 1)
