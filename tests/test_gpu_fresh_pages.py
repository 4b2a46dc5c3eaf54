"""Host-buffer queries into pages that were never touched (a fresh mapping): the library
populates them piece by piece and runs the traversal in pieces.  Records equal those of a
touched buffer at sizes around the piece and page sizes, at odd addresses, and the bytes
around the records stay as they were."""
import mmap

import numpy as np
import pytest

from portablert_gb300 import hitreg, workloads as W

pytestmark = pytest.mark.gpu

TAGS = hitreg.TAGS
PIECE = (8 << 20) // 32  # rays of 32-byte records in one piece


@pytest.fixture(scope="module")
def scene(gpu_backend):
    gpu_backend.set_tris(W.soup_tris(3, 3000))
    return gpu_backend


def _into(b, rays, addr, tags):
    lay = hitreg.layout(tags)
    b._check(b._L.prt_b200_nearest_hits(b.ctx, rays.ctypes.data, len(rays), lay.mask, lay.size,
                                        lay.offsets8(), addr))


@pytest.mark.parametrize("direct", [1, 0])
@pytest.mark.parametrize("tags", [TAGS, ("valid",)])
@pytest.mark.parametrize("n,shift", [(1, 0), (4095, 0), (4097, 4), (PIECE - 1, 0), (PIECE, 12),
                                     (PIECE + 1, 65_532), (2 * PIECE + 33, 1)])
def test_fresh_mapping(scene, n, shift, tags, direct):
    b, lay = scene, hitreg.layout(tags)
    rays = W.soup_rays(5, min(n, 5000))[np.arange(n) % min(n, 5000)]
    rays = np.ascontiguousarray(rays)
    want = np.zeros(n * lay.size, np.uint8)
    want[:] = 0  # touched
    try:
        b.set_option("host_direct", direct)
        _into(b, rays, want.ctypes.data, tags)
        room = shift + n * lay.size + 65_536
        m = mmap.mmap(-1, room)
        fresh = np.frombuffer(m, np.uint8)
        _into(b, rays, fresh.ctypes.data + shift, tags)
        assert np.array_equal(fresh[shift:shift + n * lay.size], want)
        assert not fresh[:shift].any() and not fresh[shift + n * lay.size:].any()
    finally:
        b.set_option("host_direct", 1)
