"""A host-buffer query that fails halfway may return only when nothing that it queued can still
read or write its caller's buffers, and a context may be destroyed before its batches and
servers.  Runs without a GPU, on a fake CUDA runtime whose launches fail on demand (the
library's own host code is the real one)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAILING_QUERY = """
import ctypes, mmap, sys
import numpy as np
from portablert_gb300 import _lib, hitreg

direct, launch = int(sys.argv[1]), int(sys.argv[2])
fake = ctypes.CDLL(sys.argv[3])
L = _lib.load()
h = ctypes.c_void_p()
assert L.prt_b200_create(0, ctypes.byref(h)) == 0, L.prt_b200_last_error(None)
assert L.prt_b200_set_tris(h, None, 0) == 0, L.prt_b200_last_error(h)
assert L.prt_b200_set_option(h, b"host_direct", direct) == 0
lay = hitreg.layout(hitreg.TAGS)
n = 1_100_000  # 35 MB of records: several pieces, several chunks
rays = np.ones((n, 6), np.float32)
out = mmap.mmap(-1, n * lay.size)  # never touched
addr = ctypes.addressof(ctypes.c_char.from_buffer(out))
fake.fake_pending.restype = ctypes.c_long
def query():
    return L.prt_b200_nearest_hits(h, rays.ctypes.data, n, lay.mask, lay.size, lay.offsets8(), addr)
fake.fake_fail_launch(ctypes.c_long(launch))
assert query() == 2, "the launch did not fail"
assert fake.fake_pending() == 0, "returned with work in flight"
assert query() == 0, "the context is not usable after the failure"
print("OK")
"""


@pytest.fixture(scope="module")
def fake_runtime(tmp_path_factory):
    from portablert_gb300 import build

    build.build_library()
    lib = tmp_path_factory.mktemp("fake") / "libfake_cudart.so"
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC",
                    "-I" + os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", str(lib)],
                   check=True)
    return str(lib)


def run_on_fake(fake, script, *args):
    env = dict(os.environ, LD_PRELOAD=fake, PYTHONPATH=ROOT)
    return subprocess.run([sys.executable, "-c", script, *map(str, args), fake], env=env,
                          capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("direct,launch", [(1, 1), (1, 2), (1, 4), (0, 1), (0, 3)])
def test_nothing_in_flight_after_a_failed_launch(fake_runtime, direct, launch):
    r = run_on_fake(fake_runtime, FAILING_QUERY, direct, launch)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr


LIFETIMES = """
import ctypes, sys
from portablert_gb300 import _lib
from portablert_gb300.backend import B200Backend
from portablert_gb300.batch import Batch
from portablert_gb300.serve import Server

persistent = int(sys.argv[1])
b = B200Backend(0)
b.init()
b.set_option("serve_persistent", persistent)
batches = [Batch(b), Batch(b)]
for k in batches:
    k.set_tris_dev(0, [0, 0])
server = Server(b, 0, [0, 0], 1 << 20, lanes=2)
batches[0].close()
b.shutdown()
blocks = [bytearray(256) for _ in range(4096)]  # the freed context's memory is used again
batches[1].set_tris_dev(0, [0, 0, 0])
assert batches[1].stat("n_scenes") == 2
batches[1].sync()
server.close()
batches[1].close()
b.init()
b.shutdown()
print("OK")
"""


@pytest.mark.parametrize("persistent", [0, 1])
def test_context_destroyed_before_its_batches_and_servers(fake_runtime, persistent, monkeypatch):
    monkeypatch.setenv("MALLOC_PERTURB_", "165")  # freed memory is overwritten
    r = run_on_fake(fake_runtime, LIFETIMES, persistent)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr
