"""The tree against the oracle's at the sizes where the build changes hands: one-point trees,
cells around the largest that one thread takes (32 points), around the largest that one block
takes (2048) and above it, where the cooperative levels split first."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _points(shape, coords, n, rng):
    if shape == "lattice":        # many equal coordinates and repeated points, exact sums
        x, y, z = (rng.integers(0, 12, n).astype(float) for _ in range(3))
    elif shape == "chain":        # geometric spacing: every split leaves all but a few
        x = 1.2 ** np.arange(n, dtype=float)[rng.permutation(n)]
        y, z = rng.uniform(0, 1, n), rng.uniform(0, 1, n)
    else:
        x, y, z = (rng.normal(0, 10., n) for _ in range(3))
    if coords == "flat":
        return x, y, None
    if coords == "spherical":
        z = z + 40.0
    return x, y, z


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 64, 65, 257, 2047, 2048, 2049, 9001])
@pytest.mark.parametrize("dtype,coords,split,shape", [
    ("G", "spherical", "mean", "uniform"), ("G", "flat", "mean", "lattice"),
    ("K", "3d", "middle", "uniform"), ("N", "flat", "median", "uniform"),
    ("V", "3d", "mean", "uniform"), ("N", "flat", "middle", "chain")])
def test_tree_at_block_edges(gpu_lib, dtype, coords, split, shape, n):
    if shape == "chain":
        n = min(n, 2049) // 4 + 1          # 1.2^512 is still a finite square
    rng = np.random.default_rng(n)
    x, y, z = _points(shape, coords, n, rng)
    cat = dict(x=x, y=y, z=z, w=np.ones(n) if shape == "lattice" else rng.uniform(0.5, 1.5, n),
               g1=rng.normal(0, 0.3, n), g2=rng.normal(0, 0.3, n), k=rng.normal(0, 1., n))
    f = H.gpu_field(gpu_lib, dtype, coords, cat, 0.0, 4.0, split)
    o = H.oracle_field(dtype, coords, cat, 0.0, 4.0, split)
    assert f.getNTopLevel() == o.ntop()
    a, b = f._dump(), o.dump()
    for k in ("n", "start", "depth"):
        np.testing.assert_array_equal(a[k], b[k])
    for k in ("x", "y", "z"):
        np.testing.assert_allclose(a[k], b[k], rtol=1e-12, atol=1e-12 * max(1.0, np.abs(b[k]).max()))
    # float sums of at most n terms of order 1, taken in FP64 on both sides
    np.testing.assert_allclose(a["size"], b["size"], rtol=1e-6)
    np.testing.assert_allclose(a["w"], b["w"], rtol=1e-6)
    np.testing.assert_allclose(a["d1"], b["d1"], rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(a["d2"], b["d2"], rtol=1e-5, atol=1e-6)
