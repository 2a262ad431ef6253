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
    assert nn.stat("tensor_core") == (n == 70_000)
    if n == 70_000:
        assert nn.stat("knn_tc_fallback_queries") == 3
    assert nn.stat("knn_select_fallback") == 0
    oi, od = orc.knn(X, Q, 7, metric)
    np.testing.assert_array_equal(ind, oi)
    np.testing.assert_array_equal(dist, od)


@pytest.mark.parametrize("prec", ["s", "d"])
def test_few_queries_among_equal_rows(gpu, ab, orc, prec):
    """Queries whose bound ties with more rows than a list holds: running lists for
    them alone."""
    rng = np.random.default_rng(8)
    X, Q = rows(rng, 15_000, 20, "f" if prec == "s" else "d"), None
    X[rng.choice(len(X), 6000, replace=False)] = X[0]
    Q = rows(rng, 400, 20, X.dtype)
    Q[[3, 200, 399]] = X[0]
    nn = ab.KNN(prec, metric="manhattan", algorithm="brute").fit(X)
    ind, dist = nn.kneighbors(Q, 5)
    assert 3 <= nn.stat("knn_select_fallback") < 40
    oi, od = orc.knn(X, Q, 5, "manhattan")
    np.testing.assert_array_equal(ind, oi)
    np.testing.assert_array_equal(dist, od)
