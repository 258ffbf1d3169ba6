"""GG on the sphere with a point on a pole, where FP32 can cancel the direction to another point to
nothing: at (0, 0, +-1), and at the x of cos(90 deg) in FP64, 6.1e-17.  By the walk (bin_slop), the
packed tiles, the other tile kernel (a max_sep that is no bin edge) and the allocation-free call.

As field 1 alone: x1 = y1 = 0, so the sine of the direction is 0 at both ends, both phases are
exp(-2i pi / 2) = -1, and the pair adds w0 w g0 conj(g) to xi+ and w0 w g0 g to xi- (at 6.1e-17 this holds
to a relative 1e-8: the reference's FP64 cosine is rounding of some 1e-17 there, the sine below 1e-19).
Within 1e-5, FP32 rounding of each term under 2e-6 (see test_gpu_packed.py).

Antipodal pairs have no direction either (a full-sky lattice is made of them).

Among others, and as field 2, its phase is rounding of FP32; without a shear of its own it adds nothing
but weights and counts: the oracle's sums, at the same tolerance.  With one, no pair's sum can pass
w0 w |g0| |g|."""
import ctypes
import sys

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu

X90 = np.cos(np.pi / 2)
LO, HI, NB = 4e-5, 2e-3, 5
SIZE = np.log(HI / LO) / NB
MODES = ["walk", "packed", "tiles"]
TOP = dict(min_top=0, max_top=1)


def _ring(n, north, seed):
    rng = np.random.default_rng(seed)
    th, ph = np.exp(rng.uniform(np.log(5e-5), np.log(1e-3), n)), rng.uniform(0, 2 * np.pi, n)
    return dict(x=np.sin(th) * np.cos(ph), y=np.sin(th) * np.sin(ph),
                z=np.cos(th) * (1. if north else -1.), w=rng.uniform(0.5, 1.5, n),
                g1=rng.normal(0.2, 0.3, n), g2=rng.normal(0, 0.3, n))


def _point(x0, north, g0):
    return dict(x=np.array([x0]), y=np.zeros(1), z=np.array([1. if north else -1.]), w=np.array([0.8]),
                g1=np.array([g0.real]), g2=np.array([g0.imag]))


def _bins(mode):
    bins = dict(min_sep=LO, max_sep=HI, nbins=NB, bin_size=SIZE, b=0., a=0.)
    if mode == "walk":
        bins.update(b=1e-6, a=1e-6)         # (points, not cells, as far as the phases go)
    if mode == "tiles":
        bins["max_sep"] = 0.99 * HI
    return bins


def _field(T, c):
    return H.gpu_field(T, "G", "spherical", c, 0., 0., **TOP)


@pytest.mark.parametrize("metric", ["Arc", "Euclidean"])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("x0", [0., X90, -X90])
@pytest.mark.parametrize("north", [True, False])
def test_pole_is_field_1(gpu_lib, north, x0, mode, metric):
    T = gpu_lib
    g0 = 0.4 - 0.3j
    c = _ring(700, north, 1)
    got = H.gpu_process(T, "G", metric, _bins(mode), _field(T, _point(x0, north, g0)), _field(T, c))
    assert got["npairs"].sum() == 700
    d = np.sqrt(c["x"] ** 2 + c["y"] ** 2 + (c["z"] - (1. if north else -1.)) ** 2)
    r = 2 * np.arcsin(d / 2) if metric == "Arc" else d
    k = (np.log(r / LO) / SIZE).astype(int)
    g, ww = c["g1"] + 1j * c["g2"], 0.8 * c["w"]
    for name, v in (("xi0", (g0 * g.conj()).real), ("xi2", (g0 * g).real), ("xi3", (g0 * g).imag)):
        want = np.bincount(k, weights=ww * v, minlength=NB)
        assert np.abs(got[name] - want).max() <= 1e-5 * np.abs(want).max(), (name, got[name], want)


def _noalloc(T, bins, f):
    L = T.lib()
    fn = L.tc_corr2_process_auto_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
    out = {k: np.zeros(NB) for k in H.OUT_KEYS}
    big = sys.float_info.max
    c = T.GGCorr(T.Log, LO, HI, NB, SIZE, bins["b"], bins["a"], -big, big, 0., 0., 0.,
                 *[out["xi%d" % i] for i in range(4)], out["meanr"], out["meanlogr"], out["weight"],
                 out["npairs"])
    f.getNTopLevel()
    assert fn(c._h, f._h, 0, int(T.Arc)) == 0
    return out


@pytest.mark.parametrize("g0", [0j, 0.4 - 0.3j])
@pytest.mark.parametrize("mode", MODES + ["noalloc"])
@pytest.mark.parametrize("x0", [0., X90, -X90])
@pytest.mark.parametrize("order", ["auto", "12", "21"])
def test_pole_among_others(gpu_lib, order, x0, mode, g0):
    T = gpu_lib
    if mode == "noalloc" and order != "auto":
        return
    bins = _bins("walk" if mode == "noalloc" else mode)
    ring, other = _ring(900, True, 2), _ring(500, True, 3)

    def cats(g):
        p = _point(x0, True, g)
        c = [{k: np.append(p[k], ring[k]) for k in ring}]
        return c if order == "auto" else [c[0], other] if order == "12" else [other, c[0]]
    f = [_field(T, c) for c in cats(g0)]
    got = _noalloc(T, bins, f[0]) if mode == "noalloc" else H.gpu_process(T, "G", "Arc", bins, *f)
    o = [H.oracle_field("G", "spherical", c, 0., 0., **TOP) for c in cats(0j)]
    ref = H.oracle_process("G", "Arc", bins, *o)
    if g0 == 0:
        H.assert_outputs_close(got, ref, "G", rtol=1e-5, label=f"{mode} {order}")
        return
    near = ring if order == "auto" else other
    room = 0.8 * abs(g0) * (near["w"] * np.hypot(near["g1"], near["g2"])).sum()
    tol = 1e-5 * max(np.abs(ref["xi0"]).max(), 1e-3 * ref["weight"].max())
    for k in ("xi0", "xi1", "xi2", "xi3"):
        assert np.abs(got[k] - ref[k]).sum() <= room * (1 + 1e-5) + NB * tol, k


@pytest.mark.parametrize("mode", MODES)
def test_antipodes(gpu_lib, mode):
    T = gpu_lib
    rng = np.random.default_rng(5)
    u, ph = rng.uniform(-1, 1, 300), rng.uniform(0, 2 * np.pi, 300)
    s = np.sqrt(1 - u * u)
    c = dict(x=s * np.cos(ph), y=s * np.sin(ph), z=u)
    c = {k: np.append(v, -v) for k, v in c.items()}
    c.update(w=rng.uniform(0.5, 1.5, 600), g1=rng.normal(0, 0.3, 600), g2=rng.normal(0, 0.3, 600))
    nb, lo, hi = 6, 0.05, 2.1
    size = np.log(hi / lo) / nb
    ab = 1e-6 if mode == "walk" else 0.
    bins = dict(min_sep=lo, max_sep=2.05 if mode == "tiles" else hi, nbins=nb, bin_size=size, b=ab, a=ab)
    got = H.gpu_process(T, "G", "Euclidean", bins, _field(T, c))
    ref = H.oracle_process("G", "Euclidean", bins, H.oracle_field("G", "spherical", c, 0., 0., **TOP))
    assert np.array_equal(got["npairs"], ref["npairs"])
    size = c["w"] * np.hypot(c["g1"], c["g2"])
    room = np.zeros(nb)
    room[int(np.log(2. / lo) / bins["bin_size"])] = 2 * (size[:300] * size[300:]).sum()
    tol = 1e-5 * max(np.abs(ref["xi0"]).max(), 1e-3 * ref["weight"].max())
    for k in ("xi0", "xi1", "xi2", "xi3"):
        assert np.all(np.abs(got[k] - ref[k]) <= room * (1 + 1e-5) + tol), k
