"""The slab test on centres and half extents (regular rays, FP32 nodes) must pass every box
on which the reference's slab test passes: on the CPU over the test's arithmetic restated in
numpy, on the GPU against the exhaustive search at the limits of what counts as regular."""
import numpy as np
import pytest

from portablert_gb300 import hitreg

F = np.float32
FLT_MAX = np.finfo(F).max
COORD_MAX, DIR_MAX, DIR_MIN = F(2.0 ** 67), F(2.0 ** 60), F(2.0 ** -58)


def _up(x):
    """Float64 to float32, rounded up."""
    r = x.astype(F)
    return np.where(r.astype(np.float64) < x, np.nextafter(r, F(np.inf)), r).astype(F)


def _encode(lo, hi):
    c = lo * F(0.5) + hi * F(0.5)
    c64 = c.astype(np.float64)
    e = np.maximum(_up(hi.astype(np.float64) - c64), _up(c64 - lo.astype(np.float64)))
    e = _up(e.astype(np.float64) * (1 + 2.0 ** -21))
    wide = ~((lo >= -COORD_MAX) & (hi <= COORD_MAX))
    return np.where(wide, F(0), c), np.where(wide, FLT_MAX, e)


def _passes(c, e, o, d):
    f = F(1) / d
    t = ((c - o) * f).astype(np.float64)
    g = e.astype(np.float64) * np.abs(f).astype(np.float64)
    with np.errstate(over="ignore"):
        near, far = (t - g).astype(F), (t + g).astype(F)
    tmin, tmax = np.maximum(near.max(1), F(0)), far.min(1)
    with np.errstate(over="ignore"):
        return tmin <= (tmax.astype(np.float64) * (1 + 2.0 ** -20) + 2.0 ** -120).astype(F)


def _reference(lo, hi, o, d):
    f = F(1) / d
    with np.errstate(over="ignore"):
        t1, t2 = (lo - o) * f, (hi - o) * f
    tmin, tmax = np.minimum(t1, t2).max(1), np.maximum(t1, t2).min(1)
    return (tmax >= 0) & (tmin <= tmax)


def _cases(rng, n):
    """Boxes (some flat, some enclosing a smaller box that the reference tests) and regular
    rays, many of them through a corner or along a face of the inner box."""
    scale = 2.0 ** rng.choice([-100, -40, 0, 0, 0, 20, 60], (n, 1))
    a = rng.uniform(-1, 1, (n, 3)) + rng.choice([0, 0, 1e3], (n, 1))
    w = rng.uniform(0, 1, (n, 3)) * 10.0 ** rng.uniform(-6, 0, (n, 1))
    w *= rng.random((n, 3)) > 0.15
    lo, hi = ((a - w) * scale).astype(F), ((a + w) * scale).astype(F)
    grow = np.abs(rng.normal(0, 1, (n, 3))) * w * rng.choice([0, 0, 1], (n, 1))
    olo = np.minimum(lo, ((a - w - grow) * scale).astype(F))
    ohi = np.maximum(hi, ((a + w + grow) * scale).astype(F))
    o = (rng.uniform(-3, 3, (n, 3)) * scale * 10.0 ** rng.choice([0, 0, 4], (n, 1))).astype(F)
    corner = np.where(rng.random((n, 3)) < 0.5, lo, hi).astype(np.float64)
    d = corner - o + rng.normal(0, 1, (n, 3)) * 1e-7 * scale * rng.choice([0, 1, 1e5], (n, 1))
    with np.errstate(divide="ignore", invalid="ignore"):
        d = d / np.linalg.norm(d, axis=1, keepdims=True)
    d *= 2.0 ** rng.choice([0, 0, 0, 50, -30], (n, 1))
    d = d.astype(F)
    ok = (np.abs(d) >= DIR_MIN).all(1) & (np.abs(d) <= DIR_MAX).all(1)
    ok &= (np.abs(o) <= COORD_MAX).all(1)
    return [x[ok] for x in (lo, hi, olo, ohi, o, d)]


@pytest.mark.parametrize("seed", range(6))
def test_passes_whatever_the_reference_passes(seed):
    lo, hi, olo, ohi, o, d = _cases(np.random.default_rng(seed), 200_000)
    want = _reference(lo, hi, o, d)
    assert want.sum() > 20_000 and (~want).sum() > 20_000
    c, e = _encode(olo, ohi)
    assert (_passes(c, e, o, d) | ~want).all()
    # The box of a non-finite triangle, or one past the coordinate limit.
    big = np.full_like(lo, FLT_MAX)
    c, e = _encode(-big, big)
    assert (_passes(c, e, o, d) | ~_reference(-big, big, o, d)).all()


def _scene(rng, n, scale):
    c = rng.uniform(-1, 1, (n, 1, 3))
    t = c + rng.uniform(-0.2, 0.2, (n, 3, 3))
    flat = rng.random(n) < 0.3
    t[flat, :, 1] = t[flat, :1, 1]
    return (t * scale).reshape(n, 9).astype(F)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [2.0 ** -60, 1.0, 2.0 ** 64, 2.0 ** 66.9, 2.0 ** 70])
@pytest.mark.parametrize("n", [9, 700, 5000])
def test_limits_of_regular_rays(gpu_backend, oracle_lib, scale, n):
    rng = np.random.default_rng(n)
    tris = _scene(rng, n, scale)
    m = 4096
    o = rng.uniform(-2, 2, (m, 3)) * scale
    d = rng.uniform(-1, 1, (m, 3)) * scale - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    # Whole batches at the limits, so that regular batches hold the extreme values too.
    g = (np.arange(m) // 32) % 8
    for k, v in ((1, DIR_MIN), (2, np.nextafter(DIR_MIN, F(0))), (3, F(2.0) * DIR_MIN)):
        d[g == k, k - 1] = v
    d[g == 4] *= 2.0 ** 59
    d[g == 5] *= 2.0 ** 61
    o[g == 6] *= 2.0 ** 20
    rays = np.concatenate([o, d], 1).astype(F)
    want = oracle_lib.brute_force(tris, rays)
    gpu_backend.set_tris(tris)
    got = gpu_backend.nearest_hits(rays, hitreg.TAGS)
    assert np.array_equal(got["valid"], want["valid"])
    assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
    v = want["valid"] != 0
    assert np.array_equal(got["primitive_id"][v], want["primitive_id"][v])
