"""Patch batches of so many pairs that their rows of sums pass what one launch of the walk holds
(256 MB): the pairs' counts add up to the whole catalog's (bin_slop 0, where every pair of points is
counted at its own separation), pairs are what one call per pair gives, on both sides of where
launches meet, and no more than one launch's rows stay with the corr object."""
import sys

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _corr(T, nb, lo, hi):
    o = {k: np.zeros(nb) for k in H.OUT_KEYS}
    big = sys.float_info.max
    c = T.GGCorr(T.Log, lo, hi, nb, np.log(hi / lo) / nb, 0., 0., -big, big, 0., 0., 0.,
                 *[o["xi%d" % i] for i in range(4)], o["meanr"], o["meanlogr"], o["weight"], o["npairs"])
    return c, o


@pytest.mark.parametrize("npatch,nb", [(40, 9), (850, 20)])
def test_rows_bounded(gpu_lib, npatch, nb):
    import torch
    T = gpu_lib
    rng = np.random.default_rng(npatch)
    n = 12 * npatch
    cat = dict(x=rng.uniform(0, 100., n), y=rng.uniform(0, 100., n), z=None, w=rng.uniform(0.5, 1.5, n),
               g1=rng.normal(0, 0.3, n), g2=rng.normal(0, 0.3, n))
    pid = rng.permutation(n) % npatch         # (patches all over the field: every pair is in range)
    fields = [H.gpu_field(T, "G", "flat", {k: None if v is None else np.ascontiguousarray(v[pid == p])
                                           for k, v in cat.items()}, 0., 0.) for p in range(npatch)]
    for f in fields:
        f.getNTopLevel()
    lo, hi = 1., 120.
    corr, _ = _corr(T, nb, lo, hi)
    T.TrimMemory()
    free0 = torch.cuda.mem_get_info()[0]
    pairs, res = corr.processPatches(fields, T.Euclidean)
    T.TrimMemory()
    held = free0 - torch.cuda.mem_get_info()[0]
    assert len(pairs) == npatch * (npatch + 1) // 2
    assert held <= (256 << 20) + (32 << 20), f"{held >> 20} MB held"     # (and what pieces the pool takes)
    whole, o = _corr(T, nb, lo, hi)
    whole.processAuto(H.gpu_field(T, "G", "flat", cat, 0., 0.), False, False, T.Euclidean)
    assert np.array_equal(res[:, 7].sum(0), o["npairs"])
    assert np.allclose(res[:, 0].sum(0), o["weight"], rtol=1e-6)
    step = (256 << 20) // (64 * nb)             # (pairs of one unit each that one launch holds)
    at = {0, len(pairs) - 1} | {p + d for p in range(step, len(pairs), step) for d in (-1, 0, 1)}
    for p in sorted(at | set(rng.integers(0, len(pairs), 20).tolist())):
        i, j = pairs[p]
        c, o = _corr(T, nb, lo, hi)
        if i == j:
            c.processAuto(fields[i], False, False, T.Euclidean)
        else:
            c.processCross(fields[i], fields[j], False, False, T.Euclidean)
        assert np.array_equal(res[p, 7], o["npairs"]), (i, j)
        for q, k in enumerate(("weight", "meanr", "meanlogr", "xi0", "xi1", "xi2", "xi3")):
            # (144 pairs of points: FP32 terms of under 2e-6)
            assert np.abs(res[p, q] - o[k]).max() <= 5e-6 * max(np.abs(o[k]).max(), o["weight"].max()), (i, j, k)
