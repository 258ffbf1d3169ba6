"""The packed leaf-pair tiles (exact mode; NN, scalar classes, GG on flat and spherical
coordinates) against the oracle where they can go wrong: cells of 1, 31 .. 65 leaves, self
tiles, leaves of several points and of none, lattices whose pairs crowd the bin edges (lists
that overflow), one bin, bins so narrow that a tile spans several windows of the histogram,
chords above 0.25, the ends of the range; and a tile list worked off in several drains, in
free and in fixed order.

Counts are equal.  Of the sums every term is within a few FP32 roundings (r, log r and the
phases: under 2e-6) and a tile adds up at most 64 x 2 terms per lane and bin before FP64, 8e-6
at worst: 1e-5 of the scale in all."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _catalog(coords, n, seed, layout):
    rng = np.random.default_rng(seed)
    if coords == "spherical":
        top = {"cap": 0.06, "wide": 0.9, "pole": 0.002}[layout]
        th, ph = top * np.sqrt(rng.uniform(0, 1, n)), rng.uniform(0, 2 * np.pi, n)
        x, y, z = np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)
    else:
        x, y, z = (rng.uniform(0, 30., n) for _ in range(3))
        if layout == "lattice":
            side = int(np.ceil(np.sqrt(n)))
            i = rng.permutation(n)
            x, y, z = i % side + 0.0, i // side + 0.0, z
        elif layout == "repeated":
            x, y, z = (np.round(v / 3) * 3 + rng.choice([0., 1e-3], n) for v in (x, y, z))
        z = None if coords == "flat" else z + 150.
    w = rng.uniform(0.5, 1.5, n)
    # (zero weights among coincident points, and which of two points at equal coordinates comes
    # first, are the tree's matter)
    if n > 40 and layout not in ("lattice", "repeated"):
        w[rng.integers(0, n, n // 20)] = 0.0
        w[rng.integers(0, n, n // 20)] *= -1.0
    return dict(x=x, y=y, z=z, w=w, k=rng.normal(0, 1., n), g1=rng.normal(0, 0.3, n),
                g2=rng.normal(0, 0.3, n))


# lattice edges: powers of two, moved by 1e-9 (far above FP64 rounding, far below FP32's); no pair
# at min_sep itself, where whole cells within rounding of it are the tree walk's matter
EDGES = (0.5 * (1.0 - 1e-9), 8.0 * (1.0 - 1e-9))
CASES = [
    # class, coords, metric, n1, n2, layout, nbins, (lo, hi)
    ("N", "flat", "Euclidean", 576, 0, "lattice", 4, EDGES),
    ("G", "flat", "Euclidean", 1000, 500, "lattice", 4, EDGES),
    ("K", "flat", "Euclidean", 400, 333, "lattice", 2, EDGES),
    ("G", "flat", "Euclidean", 1500, 0, "random", 1, (0.5, 40.)),
    ("N", "flat", "Euclidean", 1500, 0, "random", 50, (0.2, 35.)),
    ("G", "flat", "Euclidean", 1200, 0, "random", 40, (0.2, 35.)),
    ("K", "3d", "Euclidean", 1500, 0, "random", 35, (0.5, 45.)),
    ("N", "3d", "Euclidean", 700, 900, "repeated", 9, (1e-4, 30.)),
    ("G", "flat", "Euclidean", 900, 600, "repeated", 9, (1e-4, 30.)),
    ("K", "flat", "Euclidean", 900, 0, "repeated", 9, (2.5, 30.)),
    ("G", "spherical", "Arc", 1500, 0, "cap", 12, (0.001, 0.1)),
    ("G", "spherical", "Euclidean", 900, 700, "cap", 12, (0.001, 0.05)),
    ("G", "spherical", "Arc", 1500, 0, "wide", 6, (0.01, 1.2)),
    ("N", "spherical", "Arc", 1500, 0, "wide", 2, (0.3, 1.7)),
    ("K", "spherical", "Arc", 1500, 0, "wide", 20, (0.01, 1.7)),
    ("G", "spherical", "Arc", 800, 0, "pole", 10, (1e-5, 0.004)),
    ("NG", "spherical", "Arc", 33, 700, "cap", 6, (0.001, 0.1)),
    ("NK", "flat", "Euclidean", 65, 640, "random", 8, (0.5, 40.)),
] + [("G", "flat", "Euclidean", n, 0, "random", 3, (0.5, 45.)) for n in (2, 3, 31, 32, 33, 63, 64, 65, 129)]


TOP = dict(min_top=0, max_top=1)    # a small catalog's roots are not its leaves


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(v) for v in c[:7]))
def test_packed_tiles_vs_oracle(gpu_lib, case):
    dtype, coords, metric, n1, n2, layout, nbins, (lo, hi) = case
    T = gpu_lib
    size = np.log(hi / lo) / nbins
    bins = dict(min_sep=lo, max_sep=hi, nbins=nbins, bin_size=size, b=0.0, a=0.0)
    d1, d2 = H.kinds(dtype)
    c1 = _catalog(coords, n1, 1, layout)
    c2 = _catalog(coords, n2 or n1, 2, layout)
    f1, o1 = H.gpu_field(T, d1, coords, c1, 0., 0., **TOP), H.oracle_field(d1, coords, c1, 0., 0., **TOP)
    f2 = H.gpu_field(T, d2, coords, c2, 0., 0., **TOP) if n2 else None
    o2 = H.oracle_field(d2, coords, c2, 0., 0., **TOP) if n2 else None
    for quick in (False, True):
        got = H.gpu_process(T, dtype, metric, bins, f1, f2, quick=quick)
        ref = H.oracle_process(dtype, metric, bins, o1, o2, quick=quick)
        assert got["_stats"]["tiles"] > 0 or n1 == 2
        H.assert_outputs_close(got, ref, dtype, rtol=1e-5, label=str(case[:7]))


@pytest.mark.parametrize("fixed", [False, True])
def test_tile_list_in_several_drains(gpu_lib, fixed):
    """Tiles of at most 8 points: more than the list holds, against the default's few."""
    T = gpu_lib
    f = H.gpu_field(T, "G", "spherical", _catalog("spherical", 60000, 5, "cap"), 0., 0.)
    lo, hi, nb = 0.0005, 0.06, 15
    old = T.SetDeterministic(fixed)
    try:
        out = []
        for leaf in (8, 0):
            corr, o = _corr(T, lo, hi, nb)
            corr.setTuning(leaf, 65536)
            corr.processAuto(f, False, False, T.Arc)
            out.append(dict(o, _stats=corr.stats()))
    finally:
        T.SetDeterministic(old)
    assert out[0]["_stats"]["tiles"] > 5 << 20 > out[1]["_stats"]["tiles"]
    H.assert_outputs_close(out[0], out[1], "G", rtol=1e-5, label="drains")


def _corr(T, lo, hi, nb):
    o = {k: np.zeros(nb) for k in H.OUT_KEYS}
    big = np.finfo(float).max
    corr = T.GGCorr(T.Log, lo, hi, nb, np.log(hi / lo) / nb, 0., 0., -big, big, 0., 0., 0.,
                    *[o["xi%d" % i] for i in range(4)], o["meanr"], o["meanlogr"], o["weight"],
                    o["npairs"])
    return corr, o
