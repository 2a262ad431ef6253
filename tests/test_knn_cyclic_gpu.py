"""kNN over rows in a cyclic order (row i of class i mod C): the sampled rows meet
all classes, and a query whose bound is loose all the same (C a multiple of the
sample's step) is answered from lists with a closer bound; none needs the running
lists.  The neighbours are those of the same rows in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def data(n, nq, d, C, dtype, seed):
    rng = np.random.default_rng(seed)
    means = rng.uniform(-5, 5, (C, d))
    X = (means[np.arange(n) % C] + rng.standard_normal((n, d))).astype(dtype)
    Q = (means[rng.integers(0, C, nq)] + rng.standard_normal((nq, d))).astype(dtype)
    return rng, X, Q


def search(ab, prec, X, Q, k, metric, **options):
    nn = ab.KNN(prec, order=0, metric=metric, algorithm="brute", **options).fit(X)
    r = nn.kneighbors(Q, k)
    stats = {s: nn.stat(s) for s in ("tensor_core", "knn_tc_fallback_queries", "knn_tc_again_queries",
                                     "knn_select_fallback", "knn_select_again")}
    nn.close()
    return r, stats


@pytest.mark.parametrize("C", [7, 10, 11, 16, 19, 38, 64, 1000])
@pytest.mark.parametrize("n,nq,d,k,metric", [(200_000, 500, 64, 10, "euclidean"),
                                             (100_000, 200, 32, 100, "cosine"),
                                             (17_000, 300, 100, 256, "sqeuclidean")])
def test_tensor_core_pass(gpu, ab, C, n, nq, d, k, metric):
    _, X, Q = data(n, nq, d, C, np.float32, C)
    (ind, dist), s = search(ab, "s", X, Q, k, metric)
    assert s["tensor_core"] == 1
    assert s["knn_tc_fallback_queries"] == 0 and s["knn_select_fallback"] == 0
    (pi, pd), _ = search(ab, "s", X, Q, k, metric, precision_mode="plain")
    np.testing.assert_array_equal(ind, pi)
    np.testing.assert_array_equal(dist, pd)


@pytest.mark.parametrize("C", [2, 9, 16, 24, 64, 97])
@pytest.mark.parametrize("prec,n,nq,d,k,metric", [("s", 50_000, 400, 37, 5, "manhattan"),
                                                  ("d", 20_000, 300, 16, 40, "euclidean"),
                                                  ("s", 4_000, 40, 12, 1, "inner product"),
                                                  ("d", 9_000, 100, 20, 9, "cosine")])
def test_selection_passes(gpu, ab, orc, C, prec, n, nq, d, k, metric):
    _, X, Q = data(n, nq, d, C, np.float32 if prec == "s" else np.float64, C)
    (ind, dist), s = search(ab, prec, X, Q, k, metric)
    assert s["tensor_core"] == 0 and s["knn_select_fallback"] == 0
    oi, od = orc.knn(X, Q, k, metric)
    np.testing.assert_array_equal(ind, oi)
    np.testing.assert_array_equal(dist, od)


@pytest.mark.parametrize("prec", ["s", "d"])
def test_list_with_a_closer_bound(gpu, ab, orc, prec):
    """A cluster that the sample does not meet, far from all other rows, and as large
    as several lists: its queries take the k-th of what they listed as their next
    bound."""
    rng = np.random.default_rng(3)
    dt = np.float32 if prec == "s" else np.float64
    n, step = 40_000, 16
    X = rng.standard_normal((n, 24)).astype(dt)
    # rows that one of 16 never is, whatever its place: all but a few of each 16
    X += np.where(np.arange(n) % step < 14, 40, 0)[:, None].astype(dt)
    near = rng.choice(n, n // 10, replace=False)
    X[near] = 80 + rng.standard_normal((len(near), 24)).astype(dt)
    X[near] += (np.arange(len(near)) / 50)[:, None].astype(dt)
    Q = (80 + rng.standard_normal((200, 24))).astype(dt)
    (ind, dist), s = search(ab, prec, X, Q, 7, "manhattan")
    assert s["knn_select_fallback"] == 0
    oi, od = orc.knn(X, Q, 7, "manhattan")
    np.testing.assert_array_equal(ind, oi)
    np.testing.assert_array_equal(dist, od)
