"""The depth-first walk against the breadth-first expansion (TCGPU_WALK=0) on the same fields:
the same pairs in the same bins, and sums that agree to FP32 rounding, over the classes,
coordinates and the corners of the rule (bin_slop above 1, angle_slop binding, one bin, zero
and negative weights, brute fields, points beyond the range, a stack that is too short)."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _catalog(coords, n, seed, clump=False):
    rng = np.random.default_rng(seed)
    if coords == "spherical":
        th, ph = 0.2 * np.sqrt(rng.uniform(0, 1, n)), rng.uniform(0, 2 * np.pi, n)
        x, y, z = np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)
    else:
        x, y, z = (rng.uniform(0, 100., n) for _ in range(3))
        if clump:
            x, y, z = (np.round(v / 4) * 4 for v in (x, y, z))    # repeated points
        if coords == "flat":
            z = None
        else:
            z = z + 150.
    w = rng.uniform(0.5, 1.5, n)
    w[rng.integers(0, n, n // 20)] = 0.0
    w[rng.integers(0, n, n // 20)] *= -1.0
    return dict(x=x, y=y, z=z, w=w, k=rng.normal(0, 1., n), g1=rng.normal(0, 0.3, n),
                g2=rng.normal(0, 0.3, n))


def _bins(coords, nbins, slop, a=0.1, lo=None, hi=None):
    lo, hi = lo or (0.004 if coords == "spherical" else 1.0), hi or (0.15 if coords == "spherical" else 40.)
    size = np.log(hi / lo) / nbins
    return dict(min_sep=lo, max_sep=hi, nbins=nbins, bin_size=size, b=slop * size, a=a)


CASES = [
    # class, coords, metric, n1, n2, nbins, slop, angle_slop, clump, brute
    ("N", "flat", "Euclidean", 3000, 0, 12, 0.7, 0.1, True, False),
    ("K", "flat", "Euclidean", 2777, 0, 9, 1.0, 0.1, False, False),
    ("G", "flat", "Euclidean", 9001, 0, 20, 0.3, 0.1, False, False),
    ("G", "flat", "Euclidean", 2500, 1201, 1, 1.0, 0.1, False, False),
    ("G", "spherical", "Arc", 8000, 0, 15, 0.4, 0.1, False, False),
    ("G", "spherical", "Euclidean", 4000, 3001, 15, 0.4, 0.1, False, False),
    ("G", "spherical", "Arc", 6000, 0, 3, 1.6, 0.8, False, False),     # b above the half bin
    ("G", "spherical", "Arc", 6000, 0, 8, 0.8, 0.02, False, False),    # angle_slop binds
    ("NG", "spherical", "Arc", 900, 7000, 10, 0.5, 0.1, False, False),
    ("KG", "3d", "Euclidean", 3000, 2000, 10, 1.0, 0.1, False, False),
    ("NK", "3d", "Euclidean", 5000, 501, 10, 0.5, 0.1, True, False),
    ("V", "spherical", "Arc", 5000, 0, 10, 1.0, 0.1, False, False),
    ("T", "flat", "Euclidean", 3000, 0, 10, 1.0, 0.1, False, False),
    ("G", "3d", "Euclidean", 4000, 0, 10, 1.0, 0.1, False, False),
    ("K", "flat", "Euclidean", 1500, 700, 10, 1.0, 0.1, False, True),  # one brute field
    ("N", "spherical", "Arc", 40, 0, 5, 1.0, 0.1, False, False),
    ("N", "flat", "Euclidean", 2, 1, 5, 1.0, 0.1, False, False),
]


def _run(T, case):
    dtype, coords, metric, n1, n2, nbins, slop, a, clump, brute = case
    d1, d2 = (dtype, dtype) if len(dtype) == 1 else dtype
    bins = _bins(coords, nbins, slop, a)
    f1 = H.gpu_field(T, d1, coords, _catalog(coords, n1, 1, clump), 0.0, 0.0, brute=brute)
    f2 = H.gpu_field(T, d2, coords, _catalog(coords, n2, 2, clump), 0.0, 0.0) if n2 else None
    return lambda: H.gpu_process(T, dtype, metric, bins, f1, f2)


def _same(a, b, scale):
    assert np.array_equal(a["npairs"], b["npairs"])
    assert a["_stats"]["cell_pairs"] == b["_stats"]["cell_pairs"]
    assert a["_stats"]["accepted"] == b["_stats"]["accepted"]
    for k in H.OUT_KEYS[:-1]:
        # Sums of FP32 products with signs: FP32 rounding of at most `scale` in all.
        tol = 2e-6 * max(np.abs(b[k]).max(), scale.get(k, 0.0))
        assert np.abs(a[k] - b[k]).max() <= tol + 1e-300, k


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(v) for v in c[:8]))
def test_walk_equals_expansion(gpu_lib, monkeypatch, case):
    go = _run(gpu_lib, case)
    a, again = go(), go()
    monkeypatch.setenv("TCGPU_WALK", "0")
    b = go()
    for k in H.OUT_KEYS:
        assert np.array_equal(a[k], again[k]), k
    # The xi sums cancel: their rounding is set by the absolute sums, of the order of
    # sqrt(pairs) times the largest product (|g| <= 2, |k| <= 5, |w| <= 1.5, cells of a few).
    root = np.sqrt(np.maximum(b["npairs"], 1.).max())
    _same(a, b, {"xi%d" % i: 20. * root for i in range(4)} |
          {"weight": root, "meanr": root * 40., "meanlogr": root * 5.})


def test_short_stack_takes_the_expansion(gpu_lib, monkeypatch):
    """A walk that runs out of stack adds nothing and the call goes through the expansion."""
    go = _run(gpu_lib, CASES[2])
    a = go()
    monkeypatch.setenv("TCGPU_WALK_STACK", "160")
    b = go()
    monkeypatch.setenv("TCGPU_WALK", "0")
    c = go()
    for k in H.OUT_KEYS:
        assert np.array_equal(b[k], c[k]), k
    assert np.array_equal(a["npairs"], b["npairs"])


def test_patches_walk_equals_expansion(gpu_lib, monkeypatch):
    T = gpu_lib
    cat = _catalog("spherical", 9000, 5)
    bins = _bins("spherical", 10, 0.8)
    pid = (np.arctan2(cat["y"], cat["x"]) // 0.9).astype(int)
    fields = []
    for p in np.unique(pid):
        sel = pid == p
        fields.append(H.gpu_field(T, "G", "spherical", {k: v[sel] for k, v in cat.items()}, 0., 0.))

    def go():
        out = {k: np.zeros(10) for k in H.OUT_KEYS}
        big = np.finfo(float).max
        c = T.GGCorr(T.Log, bins["min_sep"], bins["max_sep"], 10, bins["bin_size"], bins["b"],
                     bins["a"], -big, big, 0., 0., 0., *[out[k] for k in H.OUT_KEYS])
        return c.processPatches(fields, T.Arc)
    pairs, res = go()
    assert np.array_equal(res, go()[1])       # fixed order
    monkeypatch.setenv("TCGPU_WALK", "0")
    pairs0, res0 = go()
    assert pairs == pairs0
    assert np.array_equal(res[:, 7], res0[:, 7])
    for q in range(7):
        scale = np.abs(res0[:, q]).max()
        assert np.abs(res[:, q] - res0[:, q]).max() <= 2e-6 * scale, q
