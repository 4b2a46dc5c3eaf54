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
