"""Which kernels a query launches, seen by a fake CUDA runtime: the sizes that the GPU tests of
the two passes and of packet descents use must take those routes, and stop doing so where the
rules say."""
import pytest

from routes import packet_image, two_pass_rays, warps
from test_host_failures_cpu import fake_runtime, run_on_fake  # noqa: F401 (a fixture)

SMS = 152

QUERIES = """
import ctypes, re, sys
from portablert_gb300 import _lib, hitreg
from portablert_gb300.backend import B200Backend

fmt, leaf, rays, width, height = map(int, sys.argv[1:6])
fake = ctypes.CDLL(sys.argv[6])
fake.fake_launched.restype = ctypes.c_char_p
b = B200Backend(0)
b.init()
b.set_option("leaf_size", leaf)
b.set_tris_dev(0, 0)
b.set_option("node_format", fmt)
fake.fake_forget_launched()
if rays:
    b.nearest_hits_dev(8, rays, 8)
else:
    cam = _lib.Camera()
    cam.width, cam.height, cam.sensor_size, cam.sensor_dist = width, height, 1.0, 1.0
    b.nearest_hits_camera(cam, 8)
names = fake.fake_launched().decode().split()
# k_trace8<format, count, single-triangle leaves, bounded, pass>
print(*[re.search(r"k_trace8ILi(\\d)ELb(\\d)ELb(\\d)ELb(\\d)ELi(\\d)E", n).groups() for n in names])
"""


def _launches(fake, fmt, leaf, rays=0, image=(1, 1)):
    r = run_on_fake(fake, QUERIES, fmt, leaf, rays, *image)
    assert r.returncode == 0, r.stdout + r.stderr
    return [tuple(int(c) for c in k if c.isdigit()) for k in r.stdout.strip().split(") (")]


@pytest.mark.parametrize("fmt,leaf", [(0, 1), (0, 4), (1, 1), (1, 8)])
def test_ray_buffers(fake_runtime, fmt, leaf):  # noqa: F811
    single = int(leaf == 1)
    assert _launches(fake_runtime, fmt, leaf, two_pass_rays(SMS, fmt, leaf)) == [
        (fmt, 0, single, 0, 1), (fmt, 0, single, 0, 2)]
    for rays in (1, 8 * warps(SMS) + 1, 60 * warps(SMS), two_pass_rays(SMS, fmt, leaf) - 45):
        assert _launches(fake_runtime, fmt, leaf, rays) == [(fmt, 0, single, 0, 4)], rays


@pytest.mark.parametrize("fmt,leaf", [(0, 1), (1, 4)])
def test_cameras(fake_runtime, fmt, leaf):  # noqa: F811
    single = int(leaf == 1)
    for n_tris in (0, 900):
        image = packet_image(SMS, n_tris)
        assert _launches(fake_runtime, fmt, leaf, image=image) == [(fmt, 0, single, 0, 0)]
    assert _launches(fake_runtime, fmt, leaf, image=(1021, 401)) == [(fmt, 0, single, 0, 4)]
