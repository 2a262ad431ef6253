"""k-means++ on the device at the sizes where its passes change shape: rows at
the ends of a 256-row chunk, row lengths at the ends of a 128-byte slab, 4, 6,
8 and more candidates per centre, rows whose candidates do not fit in shared
memory, many binades, leading chunks without weight -- the oracle's rows."""
import os

import numpy as np
import pytest

from test_kmeans_kpp_gpu import gmm, gpu_chosen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["s", "d"])
@pytest.mark.parametrize("n,d,k", [(255, 1, 5), (256, 31, 9), (257, 33, 60), (2049, 17, 300),
                                   (1500, 16, 1100), (300, 8300, 3)])
def test_kmeanspp_edges(gpu, ab, orc, prec, n, d, k):
    rng = np.random.default_rng(n + d)
    X = gmm(rng, n, d, 12, np.float32 if prec == "s" else np.float64)
    got, _ = gpu_chosen(ab, X, k, 3, prec, 0)
    np.testing.assert_array_equal(got, orc.kmeanspp(X, k, 3))


@pytest.mark.parametrize("prec", ["s", "d"])
@pytest.mark.parametrize("exact_draws", [False, True])
def test_kmeanspp_scales(gpu, ab, orc, prec, exact_draws):
    """Rows of scales 1e-9 .. 1e9 (a border at most chunks, sums that leave
    their binade all the time) after 3,000 copies of the first centre's row
    (chunks without weight once it is chosen), all draws also by exact sums."""
    dt = np.float32 if prec == "s" else np.float64
    rng = np.random.default_rng(8)
    X = (rng.standard_normal((9000, 6)) * 10.0 ** rng.uniform(-9, 9, (9000, 1))).astype(dt)
    X[:3000] = X[0]
    if exact_draws:
        os.environ["AOCLDA_B200_KPP_EXACT_DRAWS"] = "1"
    try:
        for seed in (1, 2, 4):
            km = ab.KMeans(25, prec, order=1, n_init=1, seed=seed)
            km.set_data(X)
            C0 = km.init_centres(25)
            km.close()
            np.testing.assert_array_equal(C0, X[orc.kmeanspp(X, 25, seed)])
    finally:
        os.environ.pop("AOCLDA_B200_KPP_EXACT_DRAWS", None)
