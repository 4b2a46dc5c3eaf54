"""Batches of scenes whose rays fit one round of small batches run as one kernel, larger ones as
two passes: each query's records must equal those of its scene alone, on both sides of the lines
(4, 8 and 16 rays per warp) and with runs that are not whole warps."""
import numpy as np
import pytest

from portablert_gb300 import _lib, hitreg, workloads as W
from portablert_gb300.batch import Batch, make_query

pytestmark = pytest.mark.gpu

TAGS = ("t", "primitive_id", "valid")


@pytest.mark.parametrize("per", [1, 4, 7, 8, 15, 16, 18])
@pytest.mark.parametrize("fmt", [0, 1])
def test_batch_graph_equals_single_scenes(gpu_backend, per, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    total = per * int(b.stat("sms")) * 32
    sizes, left = [1, 33, 500], total
    left -= sum(-(-n // 32) * 32 for n in sizes)
    sizes += [left // 64 * 32, 31, left // 2 - 77]
    sizes = [max(1, n) for n in sizes]
    scenes = [W.soup_tris(70 + i, n) for i, n in enumerate((1, 16, 300, 5000, 900, 40))]
    rays = W.soup_rays(71, 2000)
    rays[::97, 3] = 0.0
    all_rays = np.tile(rays, (-(-sum(sizes) // 2000), 1))[:sum(sizes)]
    tris = torch.from_numpy(np.concatenate(scenes).astype(np.float32)).cuda()
    off = np.concatenate([[0], np.cumsum([len(s) for s in scenes])]).astype(np.uint64)
    at = np.concatenate([[0], np.cumsum(sizes)])
    d = torch.from_numpy(np.ascontiguousarray(all_rays)).cuda()
    got = torch.full((sum(sizes), lay.size), 7, dtype=torch.uint8, device="cuda")
    want = torch.zeros_like(got)
    torch.cuda.synchronize()
    try:
        b.set_option("node_format", fmt)
        q = (_lib.Query * len(sizes))(*[
            make_query(i, d.data_ptr() + 24 * int(at[i]), n,
                       got.data_ptr() + lay.size * int(at[i]), lay.tags)
            for i, n in enumerate(sizes)])
        batch = Batch(b)
        for _ in range(2):
            batch.run_graph(tris.data_ptr(), off, q, torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            batch.sync()
        for i, s in enumerate(scenes):
            b.set_tris(s)
            b.nearest_hits_dev(d.data_ptr() + 24 * int(at[i]), sizes[i],
                               want.data_ptr() + lay.size * int(at[i]), TAGS)
            b.sync()
        assert torch.equal(got, want)
    finally:
        b.set_option("node_format", 0)
