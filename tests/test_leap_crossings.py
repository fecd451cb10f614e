"""The closed form of the DDA's repeated additions that dda_leap uses, restated
in numpy float32 against the additions themselves: same count and same bits for
increments of every kind a ray has (unit, dyadic with ties in the rounding,
near 1, huge for components of 1e-5), over every room size and many binades,
with the approximate reciprocal off by up to two units either way."""
import numpy as np
import pytest

F = np.float32


def crossings(d, a, T, most, off):
    """dda_crossings, vectorised; `off`: units added to the reciprocal."""
    f1 = d + a
    f2 = f1 + a
    i = (f2 + a) - f2
    r = ((F(1.0) / i).view(np.int32) + off).view(F)
    m = np.maximum(np.minimum(np.floor((T - f2) * r), most), F(0.0))

    def fma(x):
        return (x.astype(np.float64) * i.astype(np.float64) + f2.astype(np.float64)).astype(F)

    last = fma(m)
    over = last > T
    m = np.where(over, m - F(1.0), m)
    last = np.where(over, fma(m), last)
    nxt = last + a
    more = nxt <= T
    m = np.where(more, m + F(1.0), m)
    nxt = np.where(more, nxt + a, nxt)
    c0, c1, c2 = d <= T, f1 <= T, f2 <= T
    k = np.where(c2, m.astype(np.int64) + 3, np.where(c1, 2, np.where(c0, 1, 0)))
    return k, np.where(c2, nxt, np.where(c1, f2, np.where(c0, f1, d)))


@pytest.mark.parametrize("kind", ["random", "dyadic", "short", "odd", "axis", "unit"])
def test_leap_equals_the_additions(kind):
    rng = np.random.default_rng(7)
    n = 200000
    v = rng.normal(size=(n, 3))
    c = np.abs(v / np.linalg.norm(v, axis=1, keepdims=True)).astype(F)
    if kind == "dyadic":
        c = np.ldexp(rng.integers(1, 64, (n, 3)).astype(F), -6).astype(F)
    if kind == "axis":
        c[:] = F(1e-5)
        c[np.arange(n), rng.integers(0, 3, n)] = F(1.0)
    if kind == "unit":
        c[:] = F(1.0)
    c = np.maximum(c, F(1e-5))
    a = (F(1.0) / c).astype(F)
    if kind == "short":
        a = (a.view(np.int32) & ~0xfff).view(F)
    if kind == "odd":
        a = (a.view(np.int32) | 1).view(F)
    t0 = (2.0 ** (rng.random((n, 1)) * 11) - 1).astype(F)
    d = np.where(a < 1e4, t0 + rng.random((n, 3)).astype(F) * a, rng.random((n, 3)).astype(F) * a).astype(F)
    d[:: 17, 0] = 0.0
    side = np.array([2, 3, 4, 6, 8, 12, 16])[rng.integers(0, 7, n)]
    most = (4 * side[:, None] - 4 + rng.integers(0, 4, (n, 3))).astype(F)
    top = (((d + a).view(np.int32) & 0x7f800000) + 0x00800000).view(F)
    leave = (most.astype(np.float64) * a.astype(np.float64) + d.astype(np.float64)).astype(F)
    T = (np.minimum(leave.min(axis=1), top.min(axis=1)) * F(0.9998)).astype(F)
    for axis in range(3):
        k, e = crossings(d[:, axis], a[:, axis], T, most[:, axis], rng.integers(-2, 3, n).astype(np.int32))
        f = d[:, axis].copy()
        count = np.zeros(n, np.int64)
        for _ in range(70):
            go = f <= T
            if not go.any():
                break
            count += go
            f = np.where(go, f + a[:, axis], f)
        assert not (f <= T).any()
        np.testing.assert_array_equal(k, count)
        np.testing.assert_array_equal(e.view(np.int32), f.view(np.int32))
        assert (k <= most[:, axis]).all()          # the cube is not left
