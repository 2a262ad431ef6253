"""kNN queries that a search cannot answer from its lists are searched again, and
only they: the others' neighbours and the work for them stay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows(rng, n, d, dtype):
    means = np.random.default_rng(9).uniform(-5, 5, (30, d))
    return (means[rng.integers(0, 30, n)] + rng.standard_normal((n, d))).astype(dtype)


@pytest.mark.parametrize("dtype,n,nq,metric", [(np.float64, 10_000, 1000, "euclidean"),
                                               (np.float32, 9_000, 900, "manhattan"),
                                               (np.float64, 12_001, 70, "cosine"),
                                               (np.float32, 70_000, 300, "euclidean"),
                                               (np.float32, 70_000, 300, "cosine")])
@pytest.mark.parametrize("order", [0, 1])
def test_few_queries_without_numbers(gpu, ab, orc, dtype, n, nq, metric, order):
    rng = np.random.default_rng(n)
    X, Q = rows(rng, n, 37, dtype), rows(rng, nq, 37, dtype)
    bad = np.sort(rng.choice(nq, 3, replace=False))
    Q[bad, 5] = np.nan
    prec = "d" if dtype == np.float64 else "s"
    nn = ab.KNN(prec, order=order, metric=metric, algorithm="brute").fit(X)
    ind, dist = nn.kneighbors(Q, 7)
    # (a query that is not a number can have neighbours under the reference's cosine)
    stat = "knn_tc_fallback_queries" if nn.stat("tensor_core") else "knn_select_fallback"
    assert nn.stat("tensor_core") == (n == 70_000)
    assert nn.stat(stat) == 3
    good = np.setdiff1d(np.arange(nq), bad)
    oi, od = orc.knn(X, Q[good], 7, metric)
    np.testing.assert_array_equal(ind[good], oi)
    np.testing.assert_array_equal(dist[good], od)
    alone = nn.kneighbors(Q[bad], 7)
    np.testing.assert_array_equal(ind[bad], alone[0])
    np.testing.assert_array_equal(dist[bad], alone[1])
    assert nn.stat("knn_select_fallback") in (0, 3)
    clean = nn.kneighbors(Q[good], 7)
    np.testing.assert_array_equal(ind[good], clean[0])
    np.testing.assert_array_equal(dist[good], clean[1])
    assert nn.stat("knn_select_fallback") == 0
