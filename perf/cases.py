"""Performance cases: the work a user of this engine has it do, through its public entry
points (treecorr_gb300._treecorr), from catalog columns to finished sums.

A pass is a whole call as TreeCorr's Python layer makes it for a catalog it has not seen:
field construction (so the tree build counts), the correlation object and its process call.
Catalogs are device columns (DeviceField) except where `host` is set: then they are numpy
columns through the N/K/GField classes, as TreeCorr itself calls the module.

Outputs.  Counts (npairs, ntri, patch numbers, pair lists) are whole and returned as int64.
The other sums are FP32 products gathered in FP32 partials with wider totals; the order in
which they are gathered is left open by the interface (include/tcgpu.h, tc_corr2_set_tuning:
"the sums agree to FP32 rounding"), so they are returned as float32, the precision they
carry.  k-means centres are FP64 throughout and returned as float64.
"""
import math
import sys

import numpy as np
import torch

from treecorr_gb300 import _treecorr as T

ARCMIN = math.pi / 180.0 / 60.0
CAP_DEG2 = 1000.0          # area of the curved-sky catalogs
XI = ("xi0", "xi1", "xi2", "xi3")
KIND = {"N": 0, "K": 1, "G": 2, "Z": 3, "V": 4, "T": 5, "Q": 6}
BIG = sys.float_info.max


def listed():
    return [
        # A test or a notebook's first try: a thousand galaxies, where launches and latency
        # are all there is.
        dict(name="nn_flat_1k", op="corr2", corr="NN", coords="flat", n1=1000, n2=0, nbins=10,
             lo=1.0, hi=100.0, side=400.0, clumps=0, slop=-1.0, host=True),
        # An ordinary shear catalog of one pointing, flat sky, 20 bins 1-100 arcmin, bin_slop 1.
        dict(name="gg_flat_200k", op="corr2", corr="GG", coords="flat", n1=200_000, n2=0,
             nbins=20, lo=1.0, hi=100.0, side=1000.0, clumps=0, slop=1.0, host=True),
        # The headline: a survey's shear catalog on the curved sky at a careful bin_slop.
        dict(name="gg_sphere_10m", op="corr2", corr="GG", coords="sphere", n1=10_000_000, n2=0,
             nbins=30, lo=1.0, hi=300.0, side=0.0, clumps=0, slop=0.1, host=False),
        # The accurate mode (bin_slop 0, angle_slop 0) on a subsample, as used to check errors.
        dict(name="gg_sphere_exact_200k", op="corr2", corr="GG", coords="sphere", n1=200_003,
             n2=0, nbins=30, lo=1.0, hi=300.0, side=0.0, clumps=0, slop=0.0, host=False),
        # The accurate mode at a size where the leaf pairs are all that counts.
        dict(name="gg_sphere_exact_1m", op="corr2", corr="GG", coords="sphere", n1=1_000_000,
             n2=0, nbins=30, lo=1.0, hi=300.0, side=0.0, clumps=0, slop=0.0, host=False),
        # A scalar field in a comoving box (3-d), TreeCorr's default bin_slop.
        dict(name="kk_3d_300k", op="corr2", corr="KK", coords="3d", n1=300_017, n2=0, nbins=15,
             lo=10.0, hi=150.0, side=1000.0, clumps=0, slop=-1.0, host=False),
        # Galaxy-galaxy lensing: few lenses, many sources, default bin_slop.
        dict(name="ng_sphere_100k_2m", op="corr2", corr="NG", coords="sphere", n1=100_000,
             n2=2_000_000, nbins=20, lo=1.0, hi=200.0, side=0.0, clumps=0, slop=-1.0,
             host=False),
        # Clustering of a clumped catalog over a wide range of scales (40 bins 0.5-500 arcmin).
        dict(name="nn_clumped_2m", op="corr2", corr="NN", coords="flat", n1=2_000_000, n2=0,
             nbins=40, lo=0.5, hi=500.0, side=3000.0, clumps=100_000, slop=-1.0, host=False),
        # Jackknife covariance: every patch-pair correlation of a survey cut into patches.
        dict(name="gg_patches_1m", op="patches", n1=1_000_000, npatch=40, nbins=20, lo=1.0,
             hi=200.0, slop=-1.0),
        # Making those patches: k-means on the sky, run to its tolerance, and the assignment.
        dict(name="kmeans_2m", op="kmeans", n1=2_000_000, npatch=64),
        # Three-point shear by multipoles at the benchmark's density, bins and max_n.
        dict(name="ggg_flat_500k", op="corr3", corr="GGG", n1=500_000, n2=0, nbins=20,
             maxn=30, lo=1.0, hi=50.0, side=300.0, slop=-1.0),
        # The same, small and with bin_slop 0: a check against brute force.
        dict(name="ggg_flat_exact_5k", op="corr3", corr="GGG", n1=5000, n2=0, nbins=10,
             maxn=12, lo=1.0, hi=30.0, side=100.0, slop=0.0),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi], odd as often as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["corr2"] * 5 + ["exact"] * 2 + ["patches", "kmeans", "corr3", "corr3"])
    if what == "patches":
        return dict(op="patches", n1=_size(rng, 50_000, 1_000_000), npatch=rng.randint(8, 60),
                    nbins=rng.randint(10, 30), lo=round(rng.uniform(1.0, 3.0), 3),
                    hi=round(rng.uniform(60.0, 200.0), 2), slop=rng.choice([-1.0, 0.5]))
    if what == "kmeans":
        return dict(op="kmeans", n1=_size(rng, 20_000, 3_000_000), npatch=rng.randint(8, 150))
    if what == "corr3":
        corr = rng.choice(["GGG", "NNN", "KKK", "NGG"])
        n = _size(rng, 3000, 400_000)
        exact = corr == "GGG" and n <= 8000
        return dict(op="corr3", corr=corr, n1=n, n2=n if corr == "NGG" else 0,
                    nbins=rng.randint(5, 20), maxn=rng.randint(5, 30), lo=1.0,
                    hi=round(rng.uniform(20.0, 50.0), 2),
                    side=round(max(100.0, 300.0 * math.sqrt(n / 5e5)), 2),
                    slop=0.0 if exact else -1.0)
    coords = rng.choice(["flat", "sphere", "sphere", "3d"])
    corr = rng.choice(["NN", "KK", "GG", "GG", "NK", "NG", "KG", "VV"])
    if coords == "3d" and corr not in ("NN", "KK", "NK"):
        corr = "KK"
    if what == "exact":
        n = _size(rng, 1000, 500_000)
        slop = 0.0
    else:
        n = _size(rng, 500, 300_000 if coords == "3d" else 6_000_000)
        slop = rng.choice([-1.0, -1.0, 1.0, 0.5] + ([0.2] if n < 2_000_000 else []))
    cross = corr[0] != corr[1] or rng.random() < 0.25
    if what == "exact" and coords == "3d":
        n = min(n, 200_000)
    nbins = rng.randint(8, 40)
    lo, hi = (10.0, 150.0) if coords == "3d" else (round(rng.uniform(0.5, 3.0), 3),
                                                   round(rng.uniform(60.0, 300.0), 2))
    side = {"flat": round(20.0 * math.sqrt(max(n, 500) / 500.0) * 10.0, 1), "sphere": 0.0,
            "3d": 1000.0}[coords]
    side = min(side, 3000.0)
    return dict(op="corr2", corr=corr, coords=coords, n1=n,
                n2=_size(rng, max(500, n // 20), n) if cross else 0, nbins=nbins, lo=lo, hi=hi,
                side=side, clumps=n // 20 if coords == "flat" and rng.random() < 0.3 else 0,
                slop=slop, host=n < 300_000 and rng.random() < 0.3)


# ----------------------------------------------------------------------------------------
# Catalogs (float64 columns on the GPU, from the seed alone)

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)


def _uniform(g, n, a=0.0, b=1.0):
    return a + (b - a) * torch.rand(n, generator=g, dtype=torch.float64, device="cuda")


def _normal(g, n, s):
    return s * torch.randn(n, generator=g, dtype=torch.float64, device="cuda")


def _payload(g, kind, n, u, v, half):
    """The values of a field of this kind at plane positions u, v in [-half, half] (arcmin):
    an E-mode shear of a few long waves under shape noise, a convergence, or a vector."""
    if kind == "N":
        return []
    if kind == "K":
        return [_normal(g, n, 0.02) + 0.01 * torch.sin(u * (9.0 / half))]
    re, im = _normal(g, n, 0.25), _normal(g, n, 0.25)
    for k in range(6):
        kx, ky = (torch.rand(2, generator=g, dtype=torch.float64, device="cuda") * 40 - 20) / half
        ksq = kx * kx + ky * ky
        wave = 0.01 * torch.cos(kx * u + ky * v + k)
        re += wave * (kx * kx - ky * ky) / ksq
        im += wave * 2 * kx * ky / ksq
    return [re, im]


def _catalog(g, kind, coords, n, side=0.0, clumps=0):
    """(x, y, z or None, payload columns, w)."""
    if coords == "sphere":
        # Uniform on a 1000 deg^2 cap about (ra, dec) = (180, -30) deg.
        cmin = 1.0 - CAP_DEG2 * (math.pi / 180.0) ** 2 / (2.0 * math.pi)
        u, phi = _uniform(g, n, cmin, 1.0), _uniform(g, n, 0.0, 2.0 * math.pi)
        th = torch.acos(u)
        s = torch.sin(th)
        px, py = th / ARCMIN * torch.cos(phi), th / ARCMIN * torch.sin(phi)
        vx, vy, vz = s * torch.cos(phi), s * torch.sin(phi), u
        a = math.pi / 2 + math.radians(30.0)
        vx, vz = math.cos(a) * vx + math.sin(a) * vz, -math.sin(a) * vx + math.cos(a) * vz
        x, y, z = -vx, -vy, vz
        half = math.acos(cmin) / ARCMIN
    else:
        x, y = _uniform(g, n, 0.0, side), _uniform(g, n, 0.0, side)
        z = _uniform(g, n, 0.0, side) if coords == "3d" else None
        if clumps:
            # 40% of the points in Gaussian clumps of sigma 2 arcmin.
            cx, cy = _uniform(g, clumps, 0.0, side), _uniform(g, clumps, 0.0, side)
            m = int(0.4 * n)
            which = torch.randint(0, clumps, (m,), generator=g, device="cuda")
            x[:m] = cx[which] + _normal(g, m, 2.0)
            y[:m] = cy[which] + _normal(g, m, 2.0)
            order = torch.randperm(n, generator=g, device="cuda")
            x, y = x[order].contiguous(), y[order].contiguous()
        px, py, half = x - side / 2, y - side / 2, side / 2
    d = _payload(g, kind, n, px, py, half)
    w = torch.ones(n, dtype=torch.float64, device="cuda") if kind == "N" else _uniform(g, n, 0.5, 1.5)
    return x, y, z, d, w


def _catalogs(case, seed):
    """The catalogs of a case, one per field."""
    g = _gen(seed)
    if case["op"] == "corr2":
        a = (case["coords"], case["side"], case["clumps"])
        cats = [_catalog(g, case["corr"][0], a[0], case["n1"], a[1], a[2])]
        if case["n2"]:
            cats.append(_catalog(g, case["corr"][1], a[0], case["n2"], a[1], a[2]))
        return cats
    if case["op"] == "corr3":
        cats = [_catalog(g, case["corr"][0], "flat", case["n1"], case["side"])]
        if case["n2"]:
            cats.append(_catalog(g, case["corr"][1], "flat", case["n2"], case["side"]))
        return cats
    return [_catalog(g, "G" if case["op"] == "patches" else "N", "sphere", case["n1"])]


# ----------------------------------------------------------------------------------------
# The arguments TreeCorr's Python layer passes for a configuration

def _bins(case):
    """TreeCorr's Log binning: b = bin_slop * bin_size (default: at most 0.1), angle_slop 0.1
    (0 in the accurate mode), and the cell sizes it asks the fields for."""
    unit = ARCMIN if case.get("coords", "sphere") == "sphere" and case["op"] != "corr3" else 1.0
    lo, hi, nb, slop = case["lo"] * unit, case["hi"] * unit, case["nbins"], case["slop"]
    size = math.log(hi / lo) / nb
    b = min(size, 0.1) if slop < 0 else slop * size
    if case["op"] == "corr3":
        a = math.pi / (2 * case["maxn"] + 1) if slop != 0 else 0.0
        b1 = min(a, b)
        cells = (2 * lo * b1 / (2 + 3 * b1), hi * b1)
    else:
        a = 0.1 if slop != 0 else 0.0
        b1 = min(a, b)
        cells = (0.0, 0.0) if unit != 1.0 else (lo * b1 / (2 + 3 * b1), hi * b1)
    return dict(lo=lo, hi=hi, nb=nb, size=size, b=b, a=a, cells=cells)


def _coords(case):
    return {"flat": T.Flat, "sphere": T.Sphere, "3d": T.ThreeD}[case.get("coords", "sphere")]


def _device_field(kind, coords, cat, cells, first=0, n=None, tops=(3, 10)):
    x, y, z, d, w = cat
    n = x.numel() if n is None else n

    def p(t):
        return 0 if t is None else t.data_ptr() + 8 * first
    return T.DeviceField(KIND[kind], coords, n, p(x), p(y), p(z), p(d[0]) if d else 0,
                         p(d[1]) if len(d) > 1 else 0, p(w), 0, cells[0], cells[1], T.Mean, 0,
                         False, *tops)


def _host_field(kind, coords, cat, cells):
    x, y, z, d, w = cat
    e = np.array([])
    cls = getattr(T, kind + "Field" + {T.Flat: "Flat", T.Sphere: "Sphere", T.ThreeD: "ThreeD"}[coords])
    return cls(x, y, e if z is None else z, *d, w, e, cells[0], cells[1], T.Mean, 0, False, 3, 10)


def _xi_count(corr):
    return 0 if corr == "NN" else 1 if corr[1] in "NK" else 2 if corr[0] in "NK" else 4


def _corr2(corr, B):
    out = {k: np.zeros(B["nb"]) for k in XI[:_xi_count(corr)] + ("meanr", "meanlogr", "weight",
                                                                   "npairs")}
    e = np.array([])
    c = getattr(T, corr + "Corr")(T.Log, B["lo"], B["hi"], B["nb"], B["size"], B["b"], B["a"],
                                  -BIG, BIG, 0.0, 0.0, 0.0, *[out.get(k, e) for k in XI],
                                  out["meanr"], out["meanlogr"], out["weight"], out["npairs"])
    return c, out


def prepare(case, seed):
    cats = _catalogs(case, seed)
    state = dict(case=case, seed=int(seed), bins=None if case["op"] == "kmeans" else _bins(case))
    if case["op"] == "patches":
        # Voronoi patches of points of the catalog (uneven counts), rows ordered by patch.
        x, y, z, d, w = cats[0]
        P = torch.stack([x, y, z], 1)
        g = _gen(seed + 7)
        cen = P[torch.randperm(P.shape[0], generator=g, device="cuda")[:case["npatch"]]]
        pid = torch.cat([(c @ cen.T).argmax(1) for c in P.split(1 << 18)])
        order = torch.argsort(pid, stable=True)
        cats[0] = tuple(t[order].contiguous() for t in (x, y, z)) + (
            [t[order].contiguous() for t in d], w[order].contiguous())
        counts = torch.bincount(pid, minlength=case["npatch"]).tolist()
        state["slices"] = [(sum(counts[:i]), m) for i, m in enumerate(counts)]
    if case.get("host"):
        cats = [tuple(None if t is None else [u.cpu().numpy() for u in t] if isinstance(t, list)
                      else t.cpu().numpy() for t in c) for c in cats]
    state["cats"] = cats
    torch.cuda.synchronize()
    return state


def run(state):
    return {"corr2": _run_corr2, "patches": _run_patches, "kmeans": _run_kmeans,
            "corr3": _run_corr3}[state["case"]["op"]](state)


def _typed(out):
    return {k: np.rint(v).astype(np.int64) if k in ("npairs", "ntri") else v.astype(np.float32)
            for k, v in out.items()}


def _run_corr2(state):
    case, B = state["case"], state["bins"]
    coords = _coords(case)
    make = _host_field if case["host"] else _device_field
    f = [make(k, coords, c, B["cells"]) for k, c in zip(case["corr"], state["cats"])]
    c, out = _corr2(case["corr"], B)
    metric = T.Arc if coords == T.Sphere else T.Euclidean
    if case["n2"]:
        c.processCross(f[0], f[1], False, False, metric)
    else:
        c.processAuto(f[0], False, False, metric)
    return _typed(out)


def _run_patches(state):
    B = state["bins"]
    f = [_device_field("G", T.Sphere, state["cats"][0], B["cells"], s, n)
         for s, n in state["slices"]]
    c, _ = _corr2("GG", B)
    pairs, res = c.processPatches(f, T.Arc)
    v, cov = T.jackknife_cov(res, pairs, len(f), 2, "simple")
    table = np.zeros((len(f), len(f), 8, B["nb"]))      # pairs out of range stay zero
    i, j = np.array(pairs).T
    table[i, j] = res
    return dict(sums=table[:, :, :7].astype(np.float32),
                npairs=np.rint(table[:, :, 7]).astype(np.int64), v=v.astype(np.float32),
                cov=cov.astype(np.float32))


def _run_kmeans(state):
    n, k = state["case"]["n1"], state["case"]["npatch"]
    f = _device_field("N", T.Sphere, state["cats"][0], (0.0, math.inf),
                      tops=(min(4, k.bit_length() - 1), k.bit_length() - 1))
    cen = np.zeros((k, 3))
    f.KMeansInitTree(cen, k, state["seed"] % 100_000 + 1)
    f.KMeansRun(cen, k, 200, 1e-5, False)
    patch = np.zeros(n, dtype=np.int64)
    f.KMeansAssign(cen, k, patch)
    return dict(centres=cen, patch=patch)


def _zeta_count(corr):
    return {"NNN": 0, "KKK": 2, "NGG": 4, "GGG": 8}[corr]


def _run_corr3(state):
    case, B = state["case"], state["bins"]
    nz, mn = _zeta_count(case["corr"]), case["maxn"]
    z = ["zeta%d" % i for i in range(nz)]
    keys = z + ["meand2", "meanlogd2", "meand3", "meanlogd3", "weight", "weight_im", "ntri"]
    out = {k: np.zeros((B["nb"], B["nb"], 2 * mn + 1)) for k in keys}
    e = np.array([])
    unused = np.zeros((B["nb"], B["nb"], 2 * mn + 1))   # meand1, meanlogd1, meanu, meanv
    m = [unused, unused] + [out[k] for k in keys[nz:nz + 4]] + [unused, unused]
    c = getattr(T, case["corr"] + "Corr")(
        T.LogMultipole, B["lo"], B["hi"], B["nb"], B["size"], B["b"], B["a"], 0.0, 0.0, mn, 0.0,
        0.0, 0.0, 0.0, 0, 0.0, 0.0, -BIG, BIG, 0.0, 0.0, 0.0,
        *([out[k] for k in z] + [e] * (8 - nz)), *m, out["weight"], out["weight_im"], out["ntri"])
    f = [_device_field(k, T.Flat, cat, B["cells"]) for k, cat in zip(case["corr"], state["cats"])]
    if case["n2"]:
        c.processCross12(f[0], f[1], 1, False, False, T.Euclidean)
    else:
        c.processAuto(f[0], False, False, T.Euclidean)
    return _typed(out)


# ----------------------------------------------------------------------------------------
# What a pass cannot do without

def work(case):
    """bytes: the columns in and the results out.  flops: 80 (an FP32 curved-sky shear pair)
    per pair evaluation that the stated accuracy needs: every pair of points in range in the
    accurate mode; otherwise, per bin at separation r, the pairs of cells of size b r (or
    single points where these are sparser).  Three-point: the multipole terms of every point's
    pairs and the product of its G_n over all pairs of bins.  k-means: one distance per point
    and patch."""
    n1, n2 = case["n1"], case.get("n2", 0)
    if case["op"] == "kmeans":
        return dict(bytes=n1 * (4 * 8 + 8), flops=8.0 * n1 * case["npatch"])
    B = _bins(case)
    ncol = {"N": 0, "K": 1}
    kinds = "GG" if case["op"] == "patches" else case["corr"]
    dim = 3 if case.get("coords") == "3d" else 2
    cols = 1 + (2 if case.get("coords") == "flat" or case["op"] == "corr3" else 3)
    nbytes = 8.0 * (n1 * (cols + ncol.get(kinds[0], 2)) + n2 * (cols + ncol.get(kinds[1], 2)))
    if case["op"] == "corr3":
        area, m = case["side"] ** 2, n2 if n2 else n1
        per = m * math.pi * (B["hi"] ** 2 - B["lo"] ** 2) / area
        nn = 2 * case["maxn"] + 1
        cells = min(n1, area / max(B["b"] * B["lo"], 1e-9) ** 2)
        per = min(per, 2 * math.pi * B["nb"] * B["size"] / max(B["b"], 1e-9) ** 2)
        out = 8.0 * (_zeta_count(case["corr"]) + 7) * B["nb"] ** 2 * nn
        return dict(bytes=nbytes + out, flops=cells * (per * 16.0 * nn + 16.0 * B["nb"] ** 2 * nn))
    if case.get("coords", "sphere") == "sphere":
        area = CAP_DEG2 * (math.pi / 180.0) ** 2
    else:
        area = case["side"] ** dim
    pairs = 0.0
    for k in range(B["nb"]):
        r = B["lo"] * math.exp((k + 0.5) * B["size"])
        cell = (B["b"] * r) ** dim
        na = min(n1, area / cell) if cell > 0 else n1
        nb = min(n2 or n1, area / cell) if cell > 0 else (n2 or n1)
        shell = (2 * math.pi if dim == 2 else 4 * math.pi) * r ** dim * B["size"]
        pairs += na * nb * min(1.0, shell / area) * (1.0 if n2 else 0.5)
    out = 8.0 * 8 * B["nb"]
    if case["op"] == "patches":
        out *= case["npatch"] * 8
    return dict(bytes=nbytes + out, flops=80.0 * pairs)


# ----------------------------------------------------------------------------------------
# Brute force in 64 bits, for the cases with bin_slop 0

def exact(case, seed):
    if case["op"] == "corr2" and case["slop"] == 0.0:
        if case["n1"] * (case["n2"] or case["n1"]) > 4.5e10 or case["corr"][1] in "V":
            return None
        return _exact_corr2(case, seed)
    if case["op"] == "corr3" and case["corr"] == "GGG" and case["slop"] == 0.0 and \
            case["n1"] <= 10_000:
        return _exact_ggg(case, seed)
    return None


def _spin2(east, north, g):
    """g turned by exp(-2 i alpha), alpha the position angle of (east, north)."""
    r = torch.complex(east, north)
    return g * torch.conj(r * r) / (east * east + north * north)


def _exact_corr2(case, seed):
    """The sums over all pairs of points with lo <= r < hi, each at its own separation."""
    B, corr = _bins(case), case["corr"]
    cats = _catalogs(case, seed)
    auto = len(cats) == 1
    sphere = case["coords"] == "sphere"
    cols = []
    for kind, (x, y, z, d, w) in zip(corr, cats):
        z = torch.zeros_like(x) if z is None else z
        if sphere:
            s = torch.rsqrt(x * x + y * y + z * z)
            x, y, z = x * s, y * s, z * s
        v = w if kind == "N" else w * d[0] if kind == "K" else w * torch.complex(d[0], d[1])
        o = torch.argsort(x)
        cols.append([t[o].contiguous() for t in (x, y, z, w, v)])
    A, C = cols[0], cols[-1]
    reach = 2 * math.sin(B["hi"] / 2) if sphere else B["hi"]
    nb = B["nb"]
    nxi = _xi_count(corr)
    tot = torch.zeros(3 + nxi, nb, dtype=torch.float64, device="cuda")
    step = max(1, 40_000_000 // C[0].numel())
    for i0 in range(0, A[0].numel(), step):
        a = [t[i0:i0 + step] for t in A]
        j0 = i0 if auto else int(torch.searchsorted(C[0], a[0][:1] - reach))
        j1 = int(torch.searchsorted(C[0], a[0][-1:] + reach, right=True))
        c = [t[j0:j1] for t in C]
        if j1 <= j0:
            continue
        q = (a[0][:, None] - c[0]) ** 2 + (a[1][:, None] - c[1]) ** 2 + (a[2][:, None] - c[2]) ** 2
        near = (q < reach * reach * 1.000001) & (q > 0)
        if auto:
            near &= torch.arange(j0, j1, device="cuda") > torch.arange(
                i0, i0 + a[0].numel(), device="cuda")[:, None]
        i, j = torch.nonzero(near, as_tuple=True)
        q = q[i, j]
        r = 2 * torch.asin(q.sqrt() / 2) if sphere else q.sqrt()
        ok = (r >= B["lo"]) & (r < B["hi"])
        i, j, q, r = i[ok], j[ok], q[ok], r[ok]
        logr = r.log()
        k = ((logr - math.log(B["lo"])) / B["size"]).to(torch.int64).clamp(0, nb - 1)
        ww = a[3][i] * c[3][j]
        vals = [ww, ww * r, ww * logr]
        v1, v2 = a[4][i], c[4][j]
        if corr[1] == "G":
            x1, y1, z1, x2, y2, z2 = a[0][i], a[1][i], a[2][i], c[0][j], c[1][j], c[2][j]
            if sphere:
                east = y1 * x2 - x1 * y2
                v2 = _spin2(east, -((z1 - z2) + 0.5 * z2 * q), v2)
            else:
                v2 = _spin2(x2 - x1, y2 - y1, v2)
            if corr[0] == "G":
                v1 = _spin2(-east, -((z2 - z1) + 0.5 * z1 * q), v1) if sphere else \
                    _spin2(x2 - x1, y2 - y1, v1)
                p, m = v1 * torch.conj(v2), v1 * v2
                vals += [p.real, p.imag, m.real, m.imag]
            else:
                vals += [-(v1 * v2).real, -(v1 * v2).imag]
        elif nxi:
            vals.append(v1 * v2)
        for t, val in enumerate(vals):
            tot[t] += torch.bincount(k, weights=val, minlength=nb)
    tot = tot.cpu().numpy()
    res = dict(weight=tot[0], meanr=tot[1], meanlogr=tot[2], npairs=None)
    for t in range(nxi):
        # xi1 of GG (the odd part) has the sign of the order of each pair, which the tree sets.
        res["xi%d" % t] = None if nxi == 4 and t == 1 and auto else tot[3 + t]
    return res


def _exact_ggg(case, seed):
    """Sums over all triples by the multipoles of each point's neighbours (Porth et al.):
    G_n[k] = sum_j w_j g_j e^{-2 i phi_j} e^{i n phi_j}, W_n[k] = sum_j w_j e^{i n phi_j}, and
    their products less the terms in which both neighbours are one point."""
    B, M = _bins(case), case["maxn"]
    (x, y, _, d, w), = _catalogs(case, seed)
    n, nb, nn = x.numel(), B["nb"], 2 * case["maxn"] + 1
    wg = w * torch.complex(d[0], d[1])
    new = dict(dtype=torch.complex128, device="cuda")
    zeta = [torch.zeros(nb, nb, nn, **new) for _ in range(4)]
    weight = torch.zeros(nb, nb, nn, **new)
    means = torch.zeros(4, nb, nb, dtype=torch.float64, device="cuda")
    diag = torch.arange(nb, device="cuda")
    step = max(1, 8_000_000 // n)
    for i0 in range(0, n, step):
        rows = min(step, n - i0)
        dx, dy = x - x[i0:i0 + rows, None], y - y[i0:i0 + rows, None]
        r = torch.sqrt(dx * dx + dy * dy)
        i, j = torch.nonzero((r >= B["lo"]) & (r < B["hi"]), as_tuple=True)
        r = r[i, j]
        e = torch.complex(dx[i, j], dy[i, j]) / r
        logr = r.log()
        k = ((logr - math.log(B["lo"])) / B["size"]).to(torch.int64).clamp(0, nb - 1)
        at = i * nb + k

        def binned(v):
            t = torch.zeros(rows * nb, dtype=v.dtype, device="cuda")
            return t.index_add_(0, at, v).reshape(rows, nb)
        g = wg[j] * torch.conj(e * e)
        wj = w[j]
        W, G = {}, {}
        for m in range(-M - 1, M + 2):
            em = e ** m
            G[m] = binned(g * em)
            W[m] = binned(wj * em)
        self0 = binned(g * g * torch.conj(e * e))
        self1 = binned(g * g * e * e)
        self2 = binned((g * torch.conj(g)) * torch.conj(e * e))
        v, vg = w[i0:i0 + rows].to(torch.complex128), wg[i0:i0 + rows]

        def product(u, a, b):
            return (a * u[:, None]).T @ b
        for m in range(-M, M + 1):
            t = [product(vg, G[m - 1], G[-m - 1]), product(vg.conj(), G[m + 1], G[-m + 1]),
                 product(vg, G[m - 1], G[m + 1].conj()),
                 product(vg, G[-m + 1].conj(), G[-m - 1])]
            for q, (u, s) in enumerate(((vg, self0), (vg.conj(), self1), (vg, self2),
                                        (vg, self2))):
                t[q][diag, diag] -= (u[:, None] * s).sum(0)
                zeta[q][:, :, M + m] += t[q]
            p = product(v, W[m], W[m].conj())
            p[diag, diag] -= (v[:, None] * binned((wj * wj).to(torch.complex128))).sum(0)
            weight[:, :, M + m] += p
        sw, sr, sl = binned(wj), binned(wj * r), binned(wj * logr)
        wr, wl = binned(wj * wj * r), binned(wj * wj * logr)
        u = w[i0:i0 + rows, None]
        for q, (a, b, s) in enumerate(((sr, sw, wr), (sl, sw, wl), (sw, sr, wr), (sw, sl, wl))):
            t = (a * u).T @ b
            t[diag, diag] -= (u * s).sum(0)
            means[q] += t
    out = {"ntri": None, "weight": weight.real, "weight_im": weight.imag}
    for q in range(4):
        out["zeta%d" % (2 * q)], out["zeta%d" % (2 * q + 1)] = zeta[q].real, zeta[q].imag
    for q, name in enumerate(("meand2", "meanlogd2", "meand3", "meanlogd3")):
        full = torch.zeros(nb, nb, nn, dtype=torch.float64, device="cuda")
        full[:, :, M] = means[q]
        out[name] = full
    return {k: None if v is None else v.cpu().numpy() for k, v in out.items()}
