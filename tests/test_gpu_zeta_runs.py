"""The contraction's FP32 sums stay short for more than 32 bins (zeta.cu: RUN_MANY = 40 records to a
run, then FP64).  With weights that are whole numbers, W_0 of a vertex and the products w1 W_a W_b
are whole numbers below 2^24 / 48, so that a run of 48 terms is exact in FP32, and the sums of
products have to be the exact whole numbers.  A run of 256 passes 2^24 and rounds."""
import sys

import numpy as np
import pytest

import helpers as H
from test_gpu_multipole import MP_OUT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,w1", [(33, 1), (40, 1), (64, 3)])
def test_runs_are_short(gpu_lib, nb, w1):
    T = gpu_lib
    rng = np.random.default_rng(nb)
    n1, n2, mn, lo, hi = 1500, 39200, 2, 10., 20.
    c1 = dict(x=rng.uniform(20, 50., n1), y=rng.uniform(20, 50., n1), z=None, w=np.full(n1, float(w1)),
              g1=rng.normal(0, 0.2, n1), g2=rng.normal(0, 0.2, n1))
    c2 = dict(x=rng.uniform(0, 70., n2), y=rng.uniform(0, 70., n2), z=None, w=np.ones(n2),
              g1=rng.normal(0, 0.2, n2), g2=rng.normal(0, 0.2, n2))
    bs = np.log(hi / lo) / nb
    out = {k: np.zeros((nb, nb, 2 * mn + 1)) for k in MP_OUT}
    big = sys.float_info.max
    corr = T.GGGCorr(T.LogMultipole, lo, hi, nb, bs, 0., 0., 0., 0., mn, 0., 0., 0., 0., 0, 0., 0.,
                     -big, big, 0., 0., 0., *[out[k] for k in MP_OUT])
    f1, f2 = (H.gpu_field(T, "G", "flat", c, 0., 0.) for c in (c1, c2))
    corr.processCross12(f1, f2, 1, False, False, T.Euclidean)
    W = np.zeros((n1, nb))
    for i in range(n1):
        r = np.hypot(c2["x"] - c1["x"][i], c2["y"] - c1["y"][i])
        r = r[(r >= lo) & (r < hi)]
        W[i] = np.bincount((np.log(r / lo) / bs).astype(int).clip(0, nb - 1), minlength=nb)
    P = w1 * W.max() ** 2
    assert 48 * P <= 2 ** 24 < 256 * w1 * np.median(W[:, -1]) ** 2
    want = w1 * (W.T @ W) - np.diag(w1 * W.sum(0))
    assert np.array_equal(out["weight"][:, :, mn], want)
