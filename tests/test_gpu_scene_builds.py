"""Scene and environment builds on the GPU at the sizes where their passes
change: emissive lists around the 4096-voxel chunk and 16-voxel word of the
discovery passes, with few, many and all voxels pruned, against the
reference's sequential removal; CDFs around the 32-input chunk and the
4096-input tile, against the same sums in the same order."""
import numpy as np
import pytest

from voxeltoy_gb300 import Context, Scene
from voxeltoy_gb300 import _lib as L
from voxeltoy_gb300 import scenes as S

pytestmark = pytest.mark.gpu

PALETTE = [S.lambert(0.5), S.lambert(0.8, emission=(1.0, 2.0, 3.0)), S.lambert(0.2), S.lambert(0.1, emission=(0.0, 0.5, 0.0))]


@pytest.fixture(scope="module")
def fctx():
    c = Context()
    yield c
    c.close()


def reference_list(vox, prune):
    """Emissive voxels in voxel order, then the removal of import.cpp:180-203."""
    flat = vox.ravel()
    v = [int(i) for i in np.flatnonzero((flat == 2) | (flat == 4))]
    if not prune:
        return np.array(v, np.int32)
    p = np.pad(vox, 1)
    hidden = np.ones(vox.shape, bool)
    for d in range(3):
        for o in (0, 2):
            idx = [slice(1, -1)] * 3
            idx[d] = slice(o, p.shape[d] - 2 + o)
            hidden &= p[tuple(idx)] > 0
    keep = [not hidden.ravel()[i] for i in v]
    i = 0
    while i < len(v):
        if keep[i]:
            i += 1
            continue
        v[i], keep[i] = v[-1], keep[-1]
        v.pop()
        keep.pop()
    return np.array(v, np.int32)


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 17), (3, 5, 31), (16, 16, 16), (16, 16, 17), (1, 64, 64), (20, 33, 47),
                                   (64, 64, 65)])
@pytest.mark.parametrize("fill", ["sparse", "dense", "block"])
@pytest.mark.parametrize("prune", [False, True])
def test_emissive_lists(fctx, shape, fill, prune):
    rng = np.random.default_rng(5)
    if fill == "sparse":
        vox = (rng.random(shape) < 0.3) * rng.integers(1, 5, shape)
    elif fill == "dense":          # nearly every emissive voxel is hidden
        vox = np.where(rng.random(shape) < 0.999, rng.integers(2, 5, shape), 0)
    else:                          # a solid emissive block: hidden ones first, then shown ones at its end
        vox = np.full(shape, 2)
        vox[..., -1:] = 3
    vox = vox.astype(np.uint8)
    sc = Scene.dense(fctx, vox, PALETTE, flags=L.VT_SCENE_AUTO_EMISSIVE | (L.VT_SCENE_PRUNE_EMISSIVE if prune else 0))
    try:
        np.testing.assert_array_equal(sc.emissive(), reference_list(vox, prune))
    finally:
        sc.close()


def chunked_prefix(x):
    """FP64 prefixes: chunks of 32 left to right, chunk offsets left to right."""
    out = np.zeros(len(x) + 1)
    off = 0.0
    for c in range(0, len(x), 32):
        p = np.add.accumulate(x[c:c + 32].astype(np.float64))   # sequential
        out[c + 1:c + 1 + len(p)] = p if c == 0 else off + p
        off = p[-1] if c == 0 else off + p[-1]
    return out


@pytest.mark.parametrize("w,h", [(1, 1), (31, 3), (32, 2), (33, 65), (4095, 2), (4096, 3), (4097, 2), (9000, 2), (3, 4097)])
@pytest.mark.parametrize("kind", ["uniform", "peaked", "black_rows"])
def test_cdfs(fctx, w, h, kind):
    rng = np.random.default_rng(w * 7 + h)
    f = rng.random((h, w)).astype(np.float32)
    if kind == "peaked":
        f = (f ** 40 * np.float32(1e4)).astype(np.float32)
    if kind == "black_rows":
        f[::2] = 0.0
    cu, cv, integral = fctx.cdf_from_function(f)
    totals = np.zeros(h)
    for y in range(h):
        p = chunked_prefix(f[y])
        want = (p / p[-1]).astype(np.float32) if p[-1] > 0 else (np.arange(w + 1, dtype=np.float32) / np.float32(w))
        np.testing.assert_array_equal(cu[y], want)
        totals[y] = p[-1] / float(w)
    m = chunked_prefix(totals)
    want = (m / m[-1]).astype(np.float32) if m[-1] > 0 else (np.arange(h + 1, dtype=np.float32) / np.float32(h))
    np.testing.assert_array_equal(cv, want)
    assert np.float32(integral) == np.float32((m[-1] / float(h)) * (2.0 * 3.14159265358979323846 * 3.14159265358979323846))
