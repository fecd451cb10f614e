"""Two shortcuts of the shading code, restated in numpy float32 against what
they stand for: the tangent frame of a normal along one axis without its
normalisations, and division by a divisor known in advance by its reciprocal
and one exact remainder.  Same bits, the signs of zeros included."""
import itertools

import numpy as np
import pytest

F = np.float32
D = F(0.57735026919)


def cross(a, b):
    return [a[1] * b[2] - b[1] * a[2], a[2] * b[0] - b[2] * a[0], a[0] * b[1] - b[0] * a[1]]


def normalize(a):
    n = np.sqrt((a[0] * a[0] + a[1] * a[1]) + a[2] * a[2])
    return [c / n for c in a]


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_axis_frames_equal_the_normalised_cross_products(axis):
    for s, z0, z1 in itertools.product([F(1), F(-1)], [F(0), F(-0.0)], [F(0), F(-0.0)]):
        n = [z0, z1]
        n.insert(axis, s)
        binormal = normalize(cross(cross(n, [D, D, D]), n))
        tangent = normalize(cross(binormal, n))
        u = cross([n[1] - n[2], n[2] - n[0], n[0] - n[1]], n)
        assert np.array([F(0.70710677) * c for c in u]).tobytes() == np.array(binormal).tobytes()
        assert np.array([F(0.70710683) * c for c in cross(u, n)]).tobytes() == np.array(tangent).tobytes()


def div_known(x, c):
    # the fused operations in float64: the products of two float32 are exact
    # there, and so is the remainder; the last sum has its own rounding, which
    # differs from the fused one only next to a float32 tie, never met here
    inv = F(1) / c
    q = x * inv
    m = (q.astype(np.float64) * np.float64(c) - x.astype(np.float64)).astype(F)
    return (-m.astype(np.float64) * np.float64(inv) + q.astype(np.float64)).astype(F)


@pytest.mark.parametrize("c", [3.14159265359, 6.28318530718])
def test_division_by_pi_and_two_pi(c):
    c = F(c)
    mant = np.arange(1 << 23, dtype=np.uint32)
    for e in (24, 60, 100, 126, 127, 128, 129, 140, 200):   # biased exponents of x
        x = (mant | np.uint32(e << 23)).view(F)
        assert np.array_equal(div_known(x, c).view(np.uint32), (x / c).view(np.uint32))
    z = np.array([0.0], F)
    assert div_known(z, c).view(np.uint32)[0] == 0


@pytest.mark.parametrize("c", [1, 2, 3, 5, 64, 100, 255, 1023, 1024, 4095, 46341, 65535, (1 << 20) - 3, (1 << 20) - 2])
def test_division_of_a_voxel_by_the_resolution(c):
    x = np.arange(c, dtype=np.int64).astype(F)
    assert np.array_equal(div_known(x, F(c)).view(np.uint32), (x / F(c)).view(np.uint32))
