"""Iterations of the alternate k-means (distances with a penalty) against the oracle's, one at a time
from the oracle's centres: few patches, so that the walk takes nearly the whole tree, and many in
three dimensions, where long candidate lists last for ten levels; cells of size 0 and not, centres on
points and far from all.  The centres are FP64 means of the same cells: 1e-12 of the largest coordinate
(a cell given to another patch moves them by far more)."""
import numpy as np
import pytest

from test_gpu_walk import _catalog

import helpers as H

pytestmark = pytest.mark.gpu

CASES = [("flat", 3000, 7, 0.), ("flat", 30000, 400, 0.), ("spherical", 20000, 40, 0.), ("spherical", 9000, 900, 0.01),
         ("3d", 5000, 16, 0.), ("3d", 40000, 300, 0.), ("3d", 60000, 1500, 2.), ("3d", 2000, 17, 30.), ("3d", 300, 299, 0.)]


@pytest.mark.parametrize("coords,n,k,min_size", CASES)
@pytest.mark.parametrize("near", [1e-3, 0.3])
def test_alternate_iterations(gpu_lib, coords, n, k, min_size, near):
    T = gpu_lib
    cat = _catalog(coords, n, n + k)
    cat["w"] = np.abs(cat["w"]) + 0.1
    tops = dict(min_top=min(4, k.bit_length() - 1), max_top=k.bit_length() - 1)
    f = H.gpu_field(T, "N", coords, cat, min_size, np.inf, **tops)
    o = H.oracle_field("N", coords, cat, min_size, np.inf, **tops)
    rng = np.random.default_rng(k)
    P = np.stack([cat["x"], cat["y"]] + ([] if coords == "flat" else [cat["z"]]), 1)
    spread = (P.max(0) - P.min(0)).max()
    cen = np.ascontiguousarray(P[rng.permutation(n)[:k]] + near * spread * rng.normal(size=(k, P.shape[1])))
    for it in range(3):
        got = cen.copy()
        f.KMeansRun(got, k, 1, 0., True)
        ref, _ = o.kmeans_run(cen, 1, 0., True)
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max(), it
        cen = ref
        if len(np.unique(cen, axis=0)) < k:       # (empty patches' centres coincide: which is taken is open)
            break
