"""The G_n / W_n sums of the multipole path against direct FP64 sums over all pairs (bin_slop and
angle_slop 0: every pair on its own), at powers in one and in two rounds of 32 (max_n 5, 31, 32,
63), one bin and many, and with more records per vertex than the buffer between two
accumulations holds (4096).

z is rounded to FP32 and raised to n <= 64: an error of at most 64 x 6e-8 in phase per pair,
random in sign; the FP32 sums add at most 512 terms: 1e-5 of an array's largest value."""
import sys

import numpy as np
import pytest

import helpers as H
from test_gpu_multipole import MP_OUT

pytestmark = pytest.mark.gpu


def _cat(n, seed):
    rng = np.random.default_rng(seed)
    return dict(x=rng.uniform(0, 30., n), y=rng.uniform(0, 30., n), z=None, w=rng.uniform(0.5, 1.5, n),
                g1=rng.normal(0.05, 0.2, n), g2=rng.normal(0, 0.2, n))


@pytest.mark.parametrize("nb,mn,n1,n2", [(3, 5, 60, 700), (4, 31, 50, 600), (4, 32, 50, 600),
                                         (1, 63, 40, 500), (11, 63, 40, 500), (6, 8, 12, 11000)])
def test_sums_vs_direct(gpu_lib, nb, mn, n1, n2):
    T = gpu_lib
    c1, c2 = _cat(n1, 1), _cat(n2, 2)
    lo, hi = 1.0, 25.0
    bs = np.log(hi / lo) / nb
    out = {k: np.zeros((nb, nb, 2 * mn + 1)) for k in MP_OUT}
    big = sys.float_info.max
    corr = T.GGGCorr(T.LogMultipole, lo, hi, nb, bs, 0., 0., 0., 0., mn, 0., 0., 0., 0., 0, 0., 0.,
                     -big, big, 0., 0., 0., *[out[k] for k in MP_OUT])
    f1, f2 = (H.gpu_field(T, "G", "flat", c, 0., 0.) for c in (c1, c2))
    corr.processCross12(f1, f2, 1, False, False, T.Euclidean)
    d = (c2["x"][None] - c1["x"][:, None]) + 1j * (c2["y"][None] - c1["y"][:, None])
    r = np.abs(d)
    z = d / r
    k = np.floor(np.log(r / lo) / bs).astype(int)
    ok = (r >= lo) & (r < hi)
    wg = (c2["w"] * (c2["g1"] + 1j * c2["g2"]))[None] * np.conj(z) ** 2
    ns = np.arange(-mn - 1, mn + 2)
    G = np.zeros((n1, nb, len(ns)), complex)
    W = np.zeros((n1, nb, len(ns)), complex)
    for q, n in enumerate(ns):
        zn = z ** n
        for b in range(nb):
            m = ok & (k == b)
            G[:, b, q] = (wg * zn * m).sum(1)
            W[:, b, q] = (c2["w"][None] * zn * m).sum(1)
    w1, g1 = c1["w"], c1["w"] * (c1["g1"] + 1j * c1["g2"])
    at = lambda A, n: A[:, :, np.asarray(n) + mn + 1]
    n = np.arange(-mn, mn + 1)
    e = lambda f, A, B: np.einsum("i,ian,ibn->abn", f, A, B)
    ref = {"gam0": e(g1, at(G, n - 1), at(G, -n - 1)),
           "gam1": e(np.conj(g1), at(G, n + 1), at(G, -n + 1)),
           "gam2": e(g1, at(G, n - 1), np.conj(at(G, n + 1))),
           "gam3": e(g1, np.conj(at(G, -n + 1)), at(G, -n - 1)),
           "weight": e(w1, at(W, n), np.conj(at(W, n)))}
    npair = np.array([(ok & (k == b)).sum(1) for b in range(nb)])
    off = ~np.eye(nb, dtype=bool)
    ntri = npair @ npair.T - np.diag(npair.sum(1))
    assert np.array_equal(out["ntri"][:, :, mn], ntri)
    for name, v in ref.items():
        re = out["weight" if name == "weight" else name + "r"]
        im = out["weight_im" if name == "weight" else name + "i"]
        scale = np.abs(v).max()
        if name == "weight":                 # its self pairs are the sum of w1 w2^2
            s = np.array([(w1[:, None] * (c2["w"] ** 2)[None] * (ok & (k == b))).sum() for b in range(nb)])
            v = v - (np.eye(nb) * s)[:, :, None]
        else:                                # (the self pairs of gam turn with z: off the diagonal)
            v, re, im = v[off], re[off], im[off]
        if v.size:
            assert np.abs(re + 1j * im - v).max() <= 1e-5 * scale, name
