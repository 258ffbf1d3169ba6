"""The tree's cooperative levels against the oracle's tree: sizes around the cells that go to
one block (256 to 2048 points, by the catalog's size) and the chunks (512 to 4096), trees of more
levels than are counted at a time, and cells of which a split leaves one side empty (a centroid
outside its points: negative weights), which one block has to finish."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _compare(T, dtype, coords, cat, split):
    f = H.gpu_field(T, dtype, coords, cat, 0.0, 4.0, split)
    o = H.oracle_field(dtype, coords, cat, 0.0, 4.0, split)
    assert f.getNTopLevel() == o.ntop()
    a, b = f._dump(), o.dump()
    for k in ("n", "start", "depth"):
        np.testing.assert_array_equal(a[k], b[k])
    for k in ("x", "y", "z"):
        np.testing.assert_allclose(a[k], b[k], rtol=1e-12, atol=1e-12 * max(1.0, np.abs(b[k]).max()))
    # float sums of at most n terms of order 1, taken in FP64 on both sides
    np.testing.assert_allclose(a["size"], b["size"], rtol=1e-6)
    np.testing.assert_allclose(a["w"], b["w"], rtol=1e-6, atol=1e-6 * np.abs(b["w"]).max())
    np.testing.assert_allclose(a["d1"], b["d1"], rtol=1e-5, atol=1e-6 * np.sqrt(len(cat["x"])))
    return a


@pytest.mark.parametrize("n", [255, 256, 257, 511, 512, 513, 1025, 4097, 77825, 160001, 700001])
@pytest.mark.parametrize("dtype,coords,split", [("G", "spherical", "mean"), ("K", "flat", "middle"),
                                                ("N", "3d", "mean")])
def test_levels_by_size(gpu_lib, dtype, coords, split, n):
    rng = np.random.default_rng(n)
    x, y, z = (rng.normal(0, 10., n) for _ in range(3))
    cat = dict(x=x, y=y, z=None if coords == "flat" else z + 40., w=rng.uniform(0.5, 1.5, n),
               g1=rng.normal(0, 0.3, n), g2=rng.normal(0, 0.3, n), k=rng.normal(0, 1., n))
    _compare(gpu_lib, dtype, coords, cat, split)


@pytest.mark.parametrize("n", [2, 12, 13, 14, 25, 26, 32, 33, 104])
@pytest.mark.parametrize("dtype,coords,split", [("G", "spherical", "mean"), ("G", "flat", "median"),
                                                ("K", "3d", "middle")])
def test_one_block(gpu_lib, dtype, coords, split, n):
    # Around the cells that one thread finishes (12 points in small catalogs) and the rounds that
    # several warps share a cell in.
    rng = np.random.default_rng(n + 1000)
    x, y, z = (rng.normal(0, 10., n) for _ in range(3))
    cat = dict(x=x, y=y, z=None if coords == "flat" else z + 40., w=rng.uniform(0.5, 1.5, n),
               g1=rng.normal(0, 0.3, n), g2=rng.normal(0, 0.3, n), k=rng.normal(0, 1., n))
    _compare(gpu_lib, dtype, coords, cat, split)


def test_more_levels_than_counted(gpu_lib):
    """Weights that fall by 0.55 from point to point: every split leaves all but two."""
    n = 1000
    x = np.arange(n, dtype=float)
    perm = np.random.default_rng(3).permutation(n)
    cat = dict(x=x[perm], y=np.sin(x)[perm] * 0.1, z=None, w=(0.55 ** x)[perm], k=np.ones(n))
    a = _compare(gpu_lib, "K", "flat", cat, "mean")
    assert a["depth"].max() > 300


@pytest.mark.parametrize("n", [257, 300, 1500, 2048])
def test_one_sided_split(gpu_lib, n):
    """A root whose centroid lies outside its points."""
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 1, n)
    w = np.where(x > np.median(x), 1.0, -0.9)
    cat = dict(x=x, y=rng.uniform(0, 0.1, n), z=None, w=w, k=rng.normal(0, 1., n))
    _compare(gpu_lib, "K", "flat", cat, "mean")
