"""The inner-box test of rays with zero direction components (prt_traverse.cu, AxisRay) must pass
every box that holds a triangle box on which the reference's slab test passes: its arithmetic
restated in numpy, with origins on, beside and between faces, both zeros and denormals."""
import numpy as np
import pytest

from test_slab_margin import COORD_MAX, DIR_MIN, F, FLT_MAX, _cases, _encode

INF = F(np.inf)


def _select_min(a, b):  # portableRT's std::min / std::max: the second operand when it compares
    return np.where(b < a, b, a)


def _select_max(a, b):
    return np.where(a < b, b, a)


def _reference(lo, hi, o, d):
    with np.errstate(all="ignore"):
        f = F(1) / d
        t1, t2 = (lo - o) * f, (hi - o) * f
        near, far = _select_min(t1, t2), _select_max(t1, t2)
        tmin = _select_max(_select_max(near[:, 0], near[:, 1]), near[:, 2])
        tmax = _select_min(_select_min(far[:, 0], far[:, 1]), far[:, 2])
        return ~(tmax < 0) & ~(tmin > tmax)


def _bounds16(lo, hi):
    down = lambda x: np.where(x < 0, x.view(np.uint32) + np.uint32(0xFFFF), x.view(np.uint32))
    up = lambda x: np.where(x > 0, x.view(np.uint32) + np.uint32(0xFFFF), x.view(np.uint32))
    top = np.uint32(0xFFFF0000)
    return ((down(lo).astype(np.uint32) & top).view(F), (up(hi).astype(np.uint32) & top).view(F))


def _ray(o, d):
    """Reciprocals, the scales of near and far, and which of the ray's axes are infinite."""
    with np.errstate(all="ignore"):
        f = F(1) / d
    inf = np.isinf(f)
    past, tiny = np.abs(o) > COORD_MAX, ~inf & (np.abs(f) > F(1) / DIR_MIN)
    g = np.where(inf | past, INF, F(1))
    h = np.where(inf | past | tiny, INF, F(1))
    f = np.where(past, F(0), np.where(tiny, np.copysign(F(1) / DIR_MIN, f), f))
    return np.where(inf, np.copysign(F(1), 1 / np.where(inf, d, F(1))), f), g, h, inf


def _axis_passes(c, e, x16, o, d, x_passes):
    with np.errstate(all="ignore"):
        f, g, h, inf = _ray(o, d)
        t = ((c - o) * f).astype(np.float64)
        w = e.astype(np.float64) * np.abs(f).astype(np.float64)
        near, far = (t - w).astype(F) * g, (t + w).astype(F) * h
        outside = inf[:, 0] & ((o[:, 0] < x16[0]) | (o[:, 0] > x16[1]))
        near[:, 0] = np.where(outside, INF, near[:, 0])
        outright = inf[:, 0] & x_passes & ~(near[:, 0] > 0) & ~(far[:, 0] < 0)
        tmin = np.fmax(np.fmax.reduce(near, axis=1), F(0))
        tmax = np.fmin.reduce(far, axis=1)
        return outright | ~(tmin > (tmax.astype(np.float64) * (1 + 2.0 ** -20)
                                    + 2.0 ** -120).astype(F))


def _plain_passes(lo, hi, o, d, x_passes):
    """The same on bounds (compressed nodes)."""
    with np.errstate(all="ignore"):
        f, g, h, inf = _ray(o, d)
        t1, t2 = (lo - o) * f, (hi - o) * f
        near, far = np.fmin(t1, t2) * g, np.fmax(t1, t2) * h
        outright = inf[:, 0] & x_passes & ~(near[:, 0] > 0) & ~(far[:, 0] < 0)
        return outright | ~(np.fmax(np.fmax.reduce(near, axis=1), F(0))
                            > np.fmin.reduce(far, axis=1))


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("seed", range(6))
def test_passes_whatever_the_reference_passes(seed, odd):
    rng = np.random.default_rng(100 + seed)
    lo, hi, olo, ohi, o, d = _cases(rng, 250_000)
    n = len(lo)
    zero = rng.random((n, 3)) < 0.5
    zero[zero.all(1)] = [True, False, False]
    zero[~zero.any(1)] = [False, True, False]
    d = np.where(zero, rng.choice(np.array([0.0, -0.0, 1e-40, -1e-40], F), (n, 3)), d)
    # Origins within the box's extent, on its faces and next to them.
    at = rng.integers(0, 6, (n, 3))
    inside = (lo + (hi - lo) * rng.random((n, 3)).astype(F)).astype(F)
    beside = np.nextafter(lo, rng.choice(np.array([-np.inf, np.inf], F), (n, 3)))
    o = np.select([at == 0, at == 1, at == 2, at == 3], [lo, hi, inside, beside], o)
    shift = rng.random(n) < 0.2  # a face at zero, as on a mesh's plane of symmetry
    for k in (lo, hi, olo, ohi, o):
        k[shift, 0] -= lo[shift, 0].copy() if k is not lo else F(0)
    lo[shift, 0] = 0
    ok = (olo <= lo).all(1) & (lo <= hi).all(1) & (hi <= ohi).all(1)
    if odd:  # components outside the regular ranges, beside zeros or without
        k = rng.integers(0, 4, (n, 3))
        d = np.where(k == 0, (d * 2.0 ** rng.uniform(-125, -58, (n, 3))).astype(F), d)
        d = np.where(rng.random((n, 1)) < 0.3, (d * F(2.0 ** 63)).astype(F), d)
        o = np.where((k == 1) & (rng.random((n, 1)) < 0.3), F(2.0 ** 70) * np.sign(o), o)
        ok &= ~(np.abs(o) > COORD_MAX).all(1)
        with np.errstate(all="ignore"):
            ok &= ~np.isinf(F(1) / d).all(1)
    lo, hi, olo, ohi, o, d = (k[ok] for k in (lo, hi, olo, ohi, o, d))
    want = _reference(lo, hi, o, d)
    assert want.sum() > 20_000 and (~want).sum() > 20_000
    c, e = _encode(olo, ohi)
    x16 = _bounds16(olo[:, 0].copy(), ohi[:, 0].copy())
    # Where no lower face is at the origin's x, the x axis need not pass a box outright.
    free = o[:, 0] != lo[:, 0]
    for x_passes in (np.ones(len(lo), bool), ~free):
        assert (_axis_passes(c, e, x16, o, d, x_passes) | ~want).all()
        assert (_plain_passes(olo, ohi, o, d, x_passes) | ~want).all()
    # The box of a non-finite triangle, or one past the coordinate limit.
    big = np.full_like(lo, FLT_MAX)
    b16 = _bounds16(-big[:, 0], big[:, 0].copy())
    bc, be = _encode(-big, big)
    seen = _reference(-big, big, o, d)
    assert (_axis_passes(bc, be, b16, o, d, ~free) | ~seen).all()
    if not odd:  # It prunes: of rays that miss by a direction component that is not zero.
        missed = ~want & free & (np.abs(o - (olo + ohi) / 2) > 4 * (ohi - olo)).any(1)
        assert _axis_passes(c, e, x16, o, d, ~free)[missed].mean() < 0.2
