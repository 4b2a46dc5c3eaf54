"""What a host-buffer query does to its output pages before the device writes them, seen on a fake
CUDA runtime whose kernels write nothing: bytes outside the records stay, and records that lie
over the rays leave the rays alone, and a large output's pages are populated piece by piece while
the device has work."""
import pytest

from test_host_failures_cpu import fake_runtime, run_on_fake  # noqa: F401 (a fixture)

SCRIPT = """
import ctypes, sys
import numpy as np
from portablert_gb300 import hitreg
from portablert_gb300.backend import B200Backend

direct, n, shift = map(int, sys.argv[1:4])
b = B200Backend(0)
b.init()
b.set_option("host_direct", direct)
b.set_tris_dev(0, 0)
lay = hitreg.layout(hitreg.TAGS)
def query(rays, out):
    b._check(b._L.prt_b200_nearest_hits(b.ctx, rays, n, lay.mask, lay.size, lay.offsets8(), out))
rays = np.random.default_rng(1).random((n, 6), np.float32)
room = np.full(n * lay.size + 2 * 65536, 7, np.uint8)
query(rays.ctypes.data, room.ctypes.data + shift)
assert (room[:shift] == 7).all() and (room[shift + n * lay.size:] == 7).all()
both = np.zeros(n * lay.size // 4 + 64, np.float32)
both[16:16 + 6 * n] = rays.reshape(-1)
query(both.ctypes.data + 64, both.ctypes.data + 64)
if direct:  # (in place: no copy has brought the device's records back)
    assert np.array_equal(both[16:16 + 6 * n], rays.reshape(-1))
print("OK")
"""


@pytest.mark.parametrize("direct", [1, 0])
@pytest.mark.parametrize("n,shift", [(1, 0), (100, 4096), (5000, 65532), (30_000, 1024), (60_000, 12)])
def test_bytes_beside_the_records(fake_runtime, direct, n, shift):  # noqa: F811
    r = run_on_fake(fake_runtime, SCRIPT, direct, n, shift)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr


ORDER = """
import ctypes, mmap, sys
import numpy as np
from portablert_gb300 import hitreg
from portablert_gb300.backend import B200Backend

direct = int(sys.argv[1])
fake = ctypes.CDLL(sys.argv[2])
fake.fake_populated.restype = fake.fake_launched.restype = ctypes.c_char_p
b = B200Backend(0)
b.init()
b.set_option("host_direct", direct)
b.set_tris_dev(0, 0)
lay = hitreg.layout(hitreg.TAGS)
n = 1_500_000  # 48 MB of records
rays = np.ones((n, 6), np.float32)
out = mmap.mmap(-1, n * lay.size)  # never touched
fake.fake_forget_launched()
b._check(b._L.prt_b200_nearest_hits(b.ctx, rays.ctypes.data, n, lay.mask, lay.size, lay.offsets8(),
                                    ctypes.addressof(ctypes.c_char.from_buffer(out))))
at = [tuple(map(int, line.split())) for line in fake.fake_populated().decode().split("\\n") if line]
launches = fake.fake_launched().decode().count("\\n")
assert sum(s for _, s in at) >= n * lay.size, at
assert len(at) > 2 and launches >= len(at), (at, launches)
# At most a quarter of the pages is populated before the device has something to do, and the
# k-th piece finds at least k launches queued.
assert sum(s for k, s in at if k == 0) <= n * lay.size // 4, at
assert all(x[0] >= k for k, x in enumerate(at)), at
print("OK")
"""


@pytest.mark.parametrize("direct", [1, 0])
def test_pages_populated_while_the_device_works(fake_runtime, direct):  # noqa: F811
    r = run_on_fake(fake_runtime, ORDER, direct)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr
