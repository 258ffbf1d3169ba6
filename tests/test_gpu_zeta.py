"""The batched contraction over vertex records (zeta.cu) against the same sums taken record by
record in FP64 (a record buffer of 16 records: nearly all are contracted in place), where its
tiles and segments can go wrong: bin counts around the 4 x 2 tiles and around one block's
tiles, one bin, max_n 1 to 40, segments of one record and several segments per row range.

A factor is rounded to FP32 twice (2 x 6e-8), a product once, and a stream adds up at most
some 128 records in FP32 (128 x 6e-8 = 8e-6 at worst, were they all of one sign): 1e-5 of
an array's largest value."""
import numpy as np
import pytest

import helpers as H
from test_gpu_multipole import MP_OUT, gpu_multipole

pytestmark = pytest.mark.gpu

# nbins, max_n, points
CASES = [(1, 1, 300), (2, 3, 300), (3, 5, 6000), (4, 8, 500), (5, 40, 500), (7, 12, 500),
         (9, 2, 2000), (20, 30, 1500), (31, 4, 600), (38, 3, 600), (40, 3, 600)]


@pytest.mark.parametrize("nb,mn,n", CASES)
def test_contraction_vs_in_place(gpu_lib, monkeypatch, nb, mn, n):
    rng = np.random.default_rng(nb * 100 + mn)
    side = 40.0
    cat = dict(x=rng.uniform(0, side, n), y=rng.uniform(0, side, n), z=None,
               w=rng.uniform(0.5, 1.5, n), g1=rng.normal(0.05, 0.2, n), g2=rng.normal(0, 0.2, n))
    lo, hi = 1.0, 18.0
    bs = np.log(hi / lo) / nb
    s = dict(coords="flat", metric="Euclidean", min_sep=lo, max_sep=hi, nbins=nb, max_n=mn,
             bin_size=bs, b=min(bs, 0.1), a=np.pi / (2 * mn + 1))
    b1 = min(s["a"], s["b"])
    sizes = 2 * lo * b1 / (2 + 3 * b1), hi * b1
    out = gpu_multipole(gpu_lib, s, cat, *sizes)
    monkeypatch.setenv("TCGPU_MP_RECORD_BYTES", "0")
    ref = gpu_multipole(gpu_lib, s, cat, *sizes)
    assert np.array_equal(out["ntri"], ref["ntri"]) and ref["ntri"].sum() > 0
    for k in MP_OUT:
        assert np.abs(out[k] - ref[k]).max() <= 1e-5 * max(np.abs(ref[k]).max(), 1e-300), k
