"""The k-means tree pass with the depth-first walk, FP32 distances and batched iterations against
the oracle: short and long candidate lists, one to many patches, few large subtrees (a full
stack), repeated points and ties, coordinates far from the origin, the alternate form, and an
iteration limit inside a batch.

Assignments and iteration counts are equal; a centre is a mean of FP64 sums in another order
(1e-11 of the coordinates, as for the other runs)."""
import numpy as np
import pytest

from test_gpu_kmeans import gpu_nfield, oracle_nfield

pytestmark = pytest.mark.gpu

# coords, points, patches, top levels (min, max), alternate, iterations, layout
CASES = [
    ("flat", 30000, 1, (3, 10), False, 4, ""), ("flat", 200000, 2, (0, 1), False, 5, ""),
    ("flat", 30000, 15, (3, 10), False, 9, ""), ("flat", 30000, 17, (0, 2), False, 20, ""),
    ("flat", 60000, 300, (3, 8), False, 6, ""), ("flat", 20000, 40, (3, 6), False, 7, "lattice"),
    ("flat", 30000, 32, (3, 5), False, 8, "far"), ("flat", 300, 30, (3, 5), False, 40, ""),
    ("flat", 5000, 12, (3, 5), False, 10, "repeated"),
    ("spherical", 40000, 50, (3, 6), False, 12, ""), ("spherical", 20000, 50, (3, 6), True, 5, ""),
    ("3d", 40000, 60, (3, 6), False, 7, ""), ("3d", 20000, 20, (3, 6), True, 4, "far"),
]


@pytest.mark.parametrize("coords,n,npatch,top,alt,iters,layout", CASES)
def test_walk_vs_oracle(gpu_lib, coords, n, npatch, top, alt, iters, layout):
    rng = np.random.default_rng(n + npatch)
    x, y, z = (rng.uniform(0, 100., n) for _ in range(3))
    if layout == "lattice":
        x, y = np.arange(n) % 150 + 0.0, np.arange(n) // 150 + 0.0
    elif layout == "repeated":
        x, y = np.round(x / 10) * 10, np.round(y / 10) * 10
    elif layout == "far":
        x, y, z = x + 1e5, y - 3e5, z + 2e5
    if coords == "spherical":
        th, ph = 0.5 * np.sqrt(x / 100), y / 100 * 2 * np.pi
        x, y, z = np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)
    elif coords == "flat":
        z = None
    w = rng.uniform(0.5, 1.5, n)
    f, of = (make(coords, x, y, z, w, *top) for make in
             (lambda *a: gpu_nfield(gpu_lib, *a), oracle_nfield))
    dim = 2 if coords == "flat" else 3
    c0 = np.zeros((npatch, dim))
    f.KMeansInitRand(c0, npatch, 99)
    c = c0.copy()
    f.KMeansRun(c, npatch, iters, 0., alt)
    pat = np.zeros(n, dtype=np.int64)
    f.KMeansAssign(c, npatch, pat)
    if layout in ("lattice", "repeated"):
        # (trees of points at equal coordinates differ; the nearest centre does not)
        q = np.zeros(n, dtype=np.int64)
        gpu_lib.QuickAssign(c, npatch, x, y, np.array([]), q)
        assert np.array_equal(pat, q)
        return
    assert np.array_equal(pat, of.kmeans_assign(c))
    oc, _ = of.kmeans_run(c0, iters, 0., alt)
    np.testing.assert_allclose(c, oc, rtol=0, atol=1e-11 * np.abs(oc).max())
    if alt:
        return                      # (need not settle)
    # A tolerance that ends the run inside a batch.
    c, c1 = c0.copy(), c0.copy()
    f.KMeansRun(c, npatch, 60, 2e-3, alt)
    oc, _ = of.kmeans_run(c1, 60, 2e-3, alt)
    np.testing.assert_allclose(c, oc, rtol=0, atol=1e-11 * np.abs(oc).max())
