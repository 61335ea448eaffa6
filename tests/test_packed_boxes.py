"""The packed box test (centre and half size, kernels/traverse.cuh child_boxes and
kernels/lbvh.cu pack_axis) restated in NumPy: it may never reject a box that a
ray enters before its end, whatever the box's and the ray's scale."""
import numpy as np
import pytest

F = np.float32
EPS16 = F(1.0 + 16.0 / 16777216.0)
WIDEN = F(1.0000008)


def pack(lo, hi):
    c = (F(0.5) * lo + F(0.5) * hi).astype(F)
    exact = np.maximum(hi.astype(np.float64) - c, c.astype(np.float64) - lo)
    up = exact.astype(F)
    up = np.where(up.astype(np.float64) < exact, np.nextafter(up, F(np.inf)), up)
    h64 = up.astype(np.float64) * np.float64(EPS16)
    h = h64.astype(F)
    return c, np.where(h.astype(np.float64) < h64, np.nextafter(h, F(np.inf)), h)


def fma(a, b, c):   # a * b is exact in 64 bits
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def passes(lo, hi, o, d, tmin, tmax):
    c, h = pack(lo, hi)
    d = np.where(np.abs(d) > F(1e-24), d, np.copysign(F(1e-24), d)).astype(F)
    idir = (F(1.0) / d).astype(F)
    ulp = np.random.default_rng(1).integers(-1, 2, d.shape)   # the reciprocal is within one unit in the last place
    idir = np.where(ulp < 0, np.nextafter(idir, F(0)), np.where(ulp > 0, np.nextafter(idir, F(np.inf) * np.sign(idir)), idir))
    with np.errstate(over="ignore", invalid="ignore"):
        t = ((c - o).astype(F) * idir).astype(F)
        n = np.fmax(fma(h, -np.abs(idir), t).max(axis=1), tmin)
        f = (np.fmin(fma(h, np.abs(idir), t).min(axis=1), tmax) * WIDEN).astype(F)
    return n <= f


@pytest.mark.parametrize("scale", [1e-6, 1.0, 1e5, 1e12])
@pytest.mark.parametrize("where,flat", [("any", False), ("inside", False), ("on a face", False), ("far", False),
                                        ("any", True), ("far", True)])   # (a flat box has no inside)
def test_never_culls_an_entered_box(scale, where, flat):
    rng = np.random.default_rng(7)
    n = 200_000
    centre = rng.uniform(-1, 1, (n, 3))
    half = 10.0 ** rng.uniform(-4, -0.3, (n, 3))
    if flat:
        half[np.arange(n), rng.integers(0, 3, n)] = 0.0
    lo, hi = F((centre - half) * scale), F((centre + half) * scale)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    few = rng.random((n, 3))
    d = np.where(few < 0.15, 0.0, np.where(few < 0.3, d * 10.0 ** rng.uniform(-20, -3, (n, 3)), d))
    d[np.abs(d).max(axis=1) < 1e-3, 0] = 1.0
    d = F(d)
    target = lo + (hi.astype(np.float64) - lo) * rng.random((n, 3))      # a point of the box
    if where == "inside":
        o = lo + (hi.astype(np.float64) - lo) * rng.random((n, 3))
    elif where == "on a face":
        o = target.copy()
        k = np.arange(n), rng.integers(0, 3, n)
        o[k] = np.where(rng.random(n) < 0.5, lo[k], hi[k])
    else:
        o = target - d.astype(np.float64) * (scale * rng.uniform(0.0, 4.0 if where == "any" else 1e4, (n, 1)))
    o = F(o)
    # The interval the real ray spends in the box, in extended precision.
    L, H, O, D = (x.astype(np.longdouble) for x in (lo, hi, o, d))
    with np.errstate(divide="ignore", invalid="ignore"):
        a, b = (L - O) / D, (H - O) / D
    inside = (O >= L) & (O <= H)
    still = D == 0
    near = np.where(still, np.where(inside, -np.inf, np.inf), np.minimum(a, b)).max(axis=1)
    far = np.where(still, np.where(inside, np.inf, -np.inf), np.maximum(a, b)).min(axis=1)
    tmin = F(0.0)
    entered = (near <= far) & (far > 0)
    tmax = F(np.where(np.isfinite(near), np.maximum(near, 0), 0) * rng.uniform(1.0, 2.0, n) + scale * 1e-3)
    entered &= near <= tmax
    # A ray lying in the plane of a flat side (or on a face it leaves at once) hits no triangle of the box.
    grazing = (still & ((O == L) | (O == H))).any(axis=1)
    keep = entered & ~grazing
    assert keep.sum() > n // 50
    ok = passes(lo[keep], hi[keep], o[keep], d[keep], tmin, tmax[keep])
    assert ok.all(), f"{(~ok).sum()} of {keep.sum()} entered boxes culled"
