"""The phases z of the multipole path's pairs on flat coordinates and their powers: one vertex and one
point per bin, so that weight[a, b, n] = z_a^n conj(z_b)^n.  Against the exact phases, the rms error
may be sqrt(2) of what correctly rounded phases have when raised in FP32 the same way (below): each
part of z is rounded twice, once in d / r and once where |z| is set to 1.  (A |z| off by r's and its
reciprocal's rounding comes out at twice that: it grows with n.)"""
import sys

import numpy as np
import pytest

import helpers as H
from test_gpu_multipole import MP_OUT

pytestmark = pytest.mark.gpu

F = np.float32


def _fma(a, b, c):
    return (a.astype(float) * b.astype(float) + c.astype(float)).astype(F)


def _power(z, n):
    """z^n by multiplications in FP32, from the largest multiple of 16 below n on."""
    zr, zi = z.real.astype(F), z.imag.astype(F)
    pr, pi = np.ones_like(zr), np.zeros_like(zr)
    sr, si = zr, zi
    for _ in range(4):
        sr, si = _fma(sr, sr, -(si * si)), F(2) * sr * si
    while n > 16:
        pr, pi = _fma(pr, sr, -(pi * si)), _fma(pr, si, pi * sr)
        n -= 16
    for _ in range(n):
        pr, pi = _fma(pr, zr, -(pi * zi)), _fma(pr, zi, pi * zr)
    return pr.astype(float) + 1j * pi


@pytest.mark.parametrize("mn,ns", [(12, (6, 12)), (31, (12, 31)), (40, (31, 40))])
def test_powers_of_phases(gpu_lib, mn, ns):
    T = gpu_lib
    nb, lo, hi = 48, 1.0, 1000.0
    bs = np.log(hi / lo) / nb
    got, best = {n: [] for n in ns}, {n: [] for n in ns}
    big = sys.float_info.max
    for seed in range(12):
        rng = np.random.default_rng(seed)
        r = lo * np.exp((np.arange(nb) + rng.uniform(0.2, 0.8, nb)) * bs)
        ph = rng.uniform(0, 2 * np.pi, nb)
        x, y = (r * f(ph) for f in (np.cos, np.sin))
        x, y = x.astype(F).astype(float), y.astype(F).astype(float)     # (differences from 0 are exact)
        one = lambda n: dict(w=np.ones(n), g1=np.ones(n), g2=np.ones(n), z=None)
        f1 = H.gpu_field(T, "G", "flat", dict(one(1), x=np.zeros(1), y=np.zeros(1)), 0., 0.)
        f2 = H.gpu_field(T, "G", "flat", dict(one(nb), x=x, y=y), 0., 0.)
        out = {k: np.zeros((nb, nb, 2 * mn + 1)) for k in MP_OUT}
        corr = T.GGGCorr(T.LogMultipole, lo, hi, nb, bs, 0., 0., 0., 0., mn, 0., 0., 0., 0., 0, 0., 0.,
                         -big, big, 0., 0., 0., *[out[k] for k in MP_OUT])
        corr.processCross12(f1, f2, 1, False, False, T.Euclidean)
        off = ~np.eye(nb, dtype=bool)
        assert np.array_equal(out["ntri"][:, :, mn], off.astype(float))
        z = (x + 1j * y) / np.hypot(x, y)
        for n in ns:
            exact = np.outer(z ** n, np.conj(z) ** n)[off]
            p = _power(z, n)
            w = (out["weight"][:, :, mn + n] + 1j * out["weight_im"][:, :, mn + n])[off]
            got[n].append(np.mean(np.abs(w - exact) ** 2))
            best[n].append(np.mean(np.abs(np.outer(p, p.conj())[off] - exact) ** 2))
    for n in ns:
        ratio = np.sqrt(np.mean(got[n]) / np.mean(best[n]))
        assert ratio <= np.sqrt(2), (n, ratio)
