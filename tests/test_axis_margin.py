"""The inner-box test of rays that are not regular (prt_traverse.cu, AxisRay) must pass every box
that holds a triangle box on which the reference's slab test passes: its arithmetic restated in
numpy, with origins on, beside and between faces, both zeros, denormals, components out of the
regular ranges and origins up to the largest floats."""
import numpy as np
import pytest

from test_slab_margin import DIR_MIN, F, FLT_MAX, _cases, _encode, _passes, _up
from test_slab_margin import _reference as _regular_reference

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


def _bounds(c, e):
    """Centre and half extent to bounds, rounded outwards."""
    c, e = c.astype(np.float64), e.astype(np.float64)
    with np.errstate(over="ignore"):
        return -_up(e - c), _up(c + e)


def _passes_other(lo, hi, x16, o, d, x_passes):
    with np.errstate(all="ignore"):
        f = F(1) / d
        inf = np.isinf(f)
        g = np.where(inf, INF, F(1))
        f = np.where(inf, np.copysign(F(1), f), f)
        t1, t2 = (lo - o) * f, (hi - o) * f
        near, far = np.fmin(t1, t2) * g, np.fmax(t1, t2) * g
        if x16 is not None:
            outside = inf[:, 0] & ((o[:, 0] < x16[0]) | (o[:, 0] > x16[1]))
            near[:, 0] = np.where(outside, INF, near[:, 0])
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
        far = (2.0 ** rng.uniform(67, 127, (n, 3))).astype(F) * np.sign(o)
        o = np.where((k == 1) & (rng.random((n, 1)) < 0.3), far, o)
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
        assert (_passes_other(*_bounds(c, e), x16, o, d, x_passes) | ~want).all()
        assert (_passes_other(olo, ohi, None, o, d, x_passes) | ~want).all()  # compressed nodes
    # The box of a non-finite triangle, or one past the coordinate limit.
    big = np.full_like(lo, FLT_MAX)
    b16 = _bounds16(-big[:, 0], big[:, 0].copy())
    bc, be = _encode(-big, big)
    seen = _reference(-big, big, o, d)
    assert (_passes_other(*_bounds(bc, be), b16, o, d, ~free) | ~seen).all()
    if not odd:  # It prunes: of rays that miss by a direction component that is not zero.
        missed = ~want & free & (np.abs(o - (olo + ohi) / 2) > 4 * (ohi - olo)).any(1)
        assert _passes_other(*_bounds(c, e), x16, o, d, ~free)[missed].mean() < 0.2


@pytest.mark.parametrize("seed", range(3))
def test_long_directions_are_regular(seed):
    """Reciprocals down to the denormals: what underflow loses, the margin's 2^-120 covers."""
    rng = np.random.default_rng(200 + seed)
    lo, hi, olo, ohi, o, d = _cases(rng, 200_000)
    with np.errstate(over="ignore"):
        d = (d * 2.0 ** rng.uniform(30, 127, (len(d), 1))).astype(F)
    ok = np.isfinite(d).all(1) & (np.abs(d) >= DIR_MIN).all(1)
    lo, hi, olo, ohi, o, d = (k[ok] for k in (lo, hi, olo, ohi, o, d))
    want = _regular_reference(lo, hi, o, d)
    assert want.sum() > 10_000
    c, e = _encode(olo, ohi)
    assert (_passes(c, e, o, d) | ~want).all()
