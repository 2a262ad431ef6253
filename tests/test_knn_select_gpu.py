"""kNN with the bounds found first (the plain path's selection passes): sizes at
which the sample, the minima, the lists and the tiles change, against the
oracle, bit for bit; lists that overflow or stay short go to running lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows(rng, n, d, dtype, means):
    return (means[rng.integers(0, len(means), n)] + rng.standard_normal((n, d))).astype(dtype)


# (rows, queries, features, k): sample of all rows / every 2nd, 3rd; one row of
# queries over a tile; last slabs of 1, 4, 16 features; 2, 8 and 16 minima a
# lane; the largest k of fp64 and of fp32
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nx,nq,d,k", [(1024, 64, 16, 1), (1025, 65, 17, 16), (2047, 1, 20, 17),
                                       (3100, 129, 33, 64), (5000, 63, 4, 65),
                                       (20_011, 5, 64, 128), (9000, 3, 1, 2)])
@pytest.mark.parametrize("metric", ["euclidean", "manhattan", "inner product"])
def test_select_vs_oracle(gpu, ab, orc, dtype, nx, nq, d, k, metric):
    rng = np.random.default_rng(nx + nq + d + k)
    means = rng.uniform(-5, 5, (7, d))
    X, Q = rows(rng, nx, d, dtype, means), rows(rng, nq, d, dtype, means)
    nn = ab.KNN("d" if dtype == np.float64 else "s", order=(nx + k) % 2, metric=metric,
                algorithm="brute").fit(X)
    ind, dist = nn.kneighbors(Q, k)
    assert nn.stat("knn_select_fallback") == 0
    oi, od = orc.knn(X, Q, k, metric)
    np.testing.assert_array_equal(dist, od)
    np.testing.assert_array_equal(ind, oi)


def test_select_k256_fp32(gpu, ab, orc):
    rng = np.random.default_rng(2)
    X = rows(rng, 40_000, 24, np.float32, rng.uniform(-5, 5, (40, 24)))
    nn = ab.KNN("s", metric="sqeuclidean", algorithm="brute").fit(X)
    ind, dist = nn.kneighbors(X[:9], 256)
    assert nn.stat("knn_select_fallback") == 0
    oi, od = orc.knn(X, X[:9], 256, "sqeuclidean")
    np.testing.assert_array_equal(dist, od)
    np.testing.assert_array_equal(ind, oi)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_select_lists_that_do_not_fit(gpu, ab, orc, dtype):
    """Equal rows (every key ties with the bound) overflow the lists, NaN rows
    leave them short of k keys: running lists give the same neighbours."""
    prec = "d" if dtype == np.float64 else "s"
    rng = np.random.default_rng(4)
    X = np.tile(rng.standard_normal((3, 12)), (4000, 1)).astype(dtype)
    nn = ab.KNN(prec, metric="euclidean", algorithm="brute").fit(X)
    ind, dist = nn.kneighbors(X[:70] + dtype(0.5), 9)
    assert nn.stat("knn_select_fallback") > 0
    oi, od = orc.knn(X, X[:70] + dtype(0.5), 9)
    np.testing.assert_array_equal(dist, od)
    np.testing.assert_array_equal(ind, oi)
    X = rng.standard_normal((6000, 12)).astype(dtype)
    clean = X[:40].copy()
    X[40:] = np.nan
    nn = ab.KNN(prec, metric="euclidean", algorithm="brute").fit(X)
    ind, dist = nn.kneighbors(clean, 40)
    oi, od = orc.knn(clean, clean, 40)
    np.testing.assert_array_equal(dist, od)
    np.testing.assert_array_equal(ind, oi)
