"""Fields that one call builds side by side against the same fields built one at a time: sizes that
one block builds whole, sizes that need levels, trees with more levels than are queued at first,
more top-level cells than are read along, an empty field, a field given twice, several groups,
and fields above a group's points."""
import sys

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _cats(sizes, seed):
    rng = np.random.default_rng(seed)
    cats = []
    for k, n in enumerate(sizes):
        x, y = rng.normal(0, 10., n), rng.normal(0, 10., n)
        if k % 5 == 3:
            x = np.sign(x) * np.exp(0.5 * np.abs(x))     # long chains of uneven levels
        cats.append(dict(x=x, y=y, z=None, w=rng.uniform(0.5, 1.5, n), g1=rng.normal(0, 0.3, n),
                         g2=rng.normal(0, 0.3, n), k=rng.normal(0, 1., n)))
    return cats


def _corr(T, nb=5, lo=0.5, hi=20.):
    o = {k: np.zeros(nb) for k in H.OUT_KEYS}
    bs = np.log(hi / lo) / nb
    return T.GGCorr(T.Log, lo, hi, nb, bs, bs, 1., -sys.float_info.max, sys.float_info.max, 0., 0., 0.,
                    o["xi0"], o["xi1"], o["xi2"], o["xi3"], o["meanr"], o["meanlogr"], o["weight"],
                    o["npairs"]), o


def _same(fs, gs):
    for f, g in zip(fs, gs):
        assert f.getNTopLevel() == g.getNTopLevel()
        a, b = f._dump(), g._dump()
        for k in a:
            np.testing.assert_array_equal(a[k], b[k])


@pytest.mark.parametrize("split", ["mean", "median"])
@pytest.mark.parametrize("sizes,top", [((1, 2, 255, 256, 257, 3000, 20001, 700, 5000, 41), (3, 10)),
                                       ((7000, 30000, 9000, 12000), (11, 12)),
                                       (tuple(range(1, 140)), (3, 10))])
def test_patches_built_together(gpu_lib, sizes, top, split):
    T = gpu_lib
    make = lambda: [H.gpu_field(T, "G", "flat", c, 0.0, 4.0, split, min_top=top[0], max_top=top[1])
                    for c in _cats(sizes, len(sizes))]
    one, group = make(), make()
    for f in one:
        f.getNTopLevel()
    c, _ = _corr(T)
    d, _ = _corr(T)
    p, r = c.processPatches(one, T.Euclidean)
    q, s = d.processPatches(group + [group[0]], T.Euclidean)
    assert [x for x in q if len(one) not in x] == list(p)
    _same(one, group)


def test_empty_patch(gpu_lib):
    T = gpu_lib
    make = lambda: [H.gpu_field(T, "G", "flat", c, 0.0, 4.0) for c in _cats((500, 0, 400, 600), 4)]
    one, group = make(), make()
    for f in one:
        f.getNTopLevel()
    _corr(T)[0].processPatches(group, T.Euclidean)
    _same([one[i] for i in (0, 2, 3)], [group[i] for i in (0, 2, 3)])


@pytest.mark.parametrize("sizes", [(400, 50000), (1000, 4_200_000)])
def test_cross_built_together(gpu_lib, sizes):
    # (4.2e6 points are more than a group takes)
    T = gpu_lib
    make = lambda: [H.gpu_field(T, "G", "flat", c, 0.0, 4.0) for c in _cats(sizes, 2)]
    one, group = make(), make()
    for f in one:
        f.getNTopLevel()
    c, _ = _corr(T, lo=0.05, hi=0.2)
    c.processCross(*group, False, False, T.Euclidean)
    _same(one, group)
