"""A batch graph whose traversal pool is sized for a shallower tree than the build makes
(option pool_depth) reports it instead of answering: the pool's bounds check stops the batch and
sets the error word, which must reach the caller, once, and leave the batch usable."""
import numpy as np
import pytest

from portablert_gb300 import hitreg
from portablert_gb300._lib import PrtError
from portablert_gb300.batch import Batch, make_query

pytestmark = pytest.mark.gpu

TAGS = ("t", "primitive_id", "valid")


def _scene(n):
    """Triangles that all span the scene: every ray passes every box, so pools fill up."""
    r = np.random.default_rng(81)
    t = np.zeros((n, 3, 3))
    t[:, 0, :2] = [-5.0, -5.0]
    t[:, 1, :2] = [5.0, -5.0]
    t[:, 2, :2] = [0.0, 5.0]
    t[:, :, 2] = r.uniform(-1.0, 1.0, (n, 3))
    t[:, :, :2] += r.uniform(-0.5, 0.5, (n, 3, 2))
    return t.reshape(n, 9).astype(np.float32)


@pytest.mark.parametrize("leaf,fmt", [(1, 0), (4, 0), (1, 1)])
@pytest.mark.parametrize("n_rays", [60_000, 200_000])  # one kernel, two passes
def test_overflow_is_reported(gpu_backend, n_rays, leaf, fmt):
    import torch

    b, lay = gpu_backend, hitreg.layout(TAGS)
    n = 100_000 * leaf
    tris = torch.from_numpy(_scene(n)).cuda()
    r = np.random.default_rng(82)
    rays = np.zeros((512, 6), np.float32)
    rays[:, :2] = r.uniform(-0.5, 0.5, (512, 2))
    rays[:, 2] = -10.0
    rays[:, 3:5] = r.uniform(-0.01, 0.01, (512, 2))
    rays[:, 5] = 1.0
    rays = torch.from_numpy(rays).cuda()
    far = rays[:1].repeat(n_rays - 512, 1)  # the other rays miss the scene's box at once
    far[:, 0] = 100.0
    rays = torch.cat([rays, far]).contiguous()
    rec = torch.zeros(n_rays * lay.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    batch = Batch(b)
    try:
        b.set_option("leaf_size", leaf)
        b.set_option("node_format", fmt)
        b.set_option("collapse_cost", 0)  # full nodes: eight pushes for one pop
        q = [make_query(0, rays.data_ptr(), n_rays, rec.data_ptr(), TAGS)]
        b.set_option("pool_depth", 0)
        batch.run_graph(tris.data_ptr(), [0, n], q)
        batch.sync()
        want = rec.clone()
        assert batch.stat("depth") >= 5
        b.set_option("pool_depth", 1)
        batch.run_graph(tris.data_ptr(), [0, n], q)
        with pytest.raises(PrtError) as e:
            batch.sync()
        assert e.value.code == 5  # PRT_ERR_DEVICE
        b.set_option("pool_depth", 0)
        rec.zero_()
        torch.cuda.synchronize()
        batch.run_graph(tris.data_ptr(), [0, n], q)
        batch.sync()
        assert torch.equal(rec, want)
    finally:
        b.set_option("pool_depth", 0)
        b.set_option("collapse_cost", 1)
        b.set_option("leaf_size", 1)
        b.set_option("node_format", 0)
        batch.close()
