"""Queries and rows that are not numbers: a query with fewer than k rows at a
distance that is a number ends in index -1 at distance +inf, as the oracle's,
and what reads neighbours (votes, means, probed lists) passes over them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def data(n, nq, d, dtype, seed):
    rng = np.random.default_rng(seed)
    X, Q = rng.standard_normal((n, d)).astype(dtype), rng.standard_normal((nq, d)).astype(dtype)
    bad = np.sort(rng.choice(nq, 3, replace=False))
    Q[bad, d // 2] = np.nan
    return X, Q, bad


# (one search of small lists, one whose rows are too few for them, tensor cores)
@pytest.mark.parametrize("dtype,n,nq,k", [(np.float64, 6000, 300, 7), (np.float32, 6000, 300, 7),
                                          (np.float64, 90, 20, 50), (np.float32, 40_000, 260, 9)])
@pytest.mark.parametrize("metric", ["euclidean", "manhattan", "cosine", "inner product"])
@pytest.mark.parametrize("order", [0, 1])
def test_neighbours(gpu, ab, orc, dtype, n, nq, k, metric, order):
    X, Q, bad = data(n, nq, 24, dtype, n + k)
    nn = ab.KNN("d" if dtype == np.float64 else "s", order=order, metric=metric,
                algorithm="brute").fit(X)
    nn.kneighbors(X[:nq], k + 1)  # buffers that have held something else
    ind, dist = nn.kneighbors(Q, k)
    oi, od = orc.knn(X, Q, k, metric)
    assert (oi[bad] == -1).all()
    np.testing.assert_array_equal(ind, oi)
    np.testing.assert_array_equal(dist, od)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_rows_that_are_not_numbers(gpu, ab, orc, dtype):
    X, Q, _ = data(3000, 70, 12, dtype, 3)
    X[5:] = np.nan
    nn = ab.KNN("d" if dtype == np.float64 else "s", algorithm="brute").fit(X)
    ind, dist = nn.kneighbors(Q, 9)
    oi, od = orc.knn(X, Q, 9)
    np.testing.assert_array_equal(ind, oi)
    np.testing.assert_array_equal(dist, od)


@pytest.mark.parametrize("weights", ["uniform", "distance"])
def test_votes_and_means(gpu, ab, weights):
    X, Q, bad = data(5000, 200, 16, np.float64, 4)
    rng = np.random.default_rng(4)
    y, t = rng.integers(0, 5, len(X)), rng.standard_normal(len(X))
    nn = ab.KNN("d", number_of_neighbors=6, weights=weights, algorithm="brute").fit(X, y, t)
    nn.kneighbors(X[:200], 11)
    good = np.setdiff1d(np.arange(len(Q)), bad)
    lab, pr, reg = nn.predict(Q), nn.predict_proba(Q), nn.predict_reg(Q)
    np.testing.assert_array_equal(lab[good], nn.predict(Q[good]))
    np.testing.assert_array_equal(pr[good], nn.predict_proba(Q[good]))
    np.testing.assert_array_equal(reg[good], nn.predict_reg(Q[good]))
    assert np.isnan(reg[bad]).all()


@pytest.mark.parametrize("prec", ["s", "d"])
def test_ivf(gpu, ab, prec):
    X, Q, bad = data(5000, 60, 12, np.float32 if prec == "s" else np.float64, 5)
    h = ab.ApproxNN(prec, order=ab.ROW_MAJOR, n_list=16, n_probe=4, seed=1)
    h.set_training_data(X).train_and_add()
    good = np.setdiff1d(np.arange(len(Q)), bad)
    want = h.kneighbors(Q[good], 6)
    for _ in range(2):
        ind, dist = h.kneighbors(Q, 6)
        assert (ind[bad] == -1).all() and np.isposinf(dist[bad]).all()
        np.testing.assert_array_equal(ind[good], want[0])
        np.testing.assert_array_equal(dist[good], want[1])
        h.add(Q)  # 3 rows of it in no list's neighbourhood; the others are found
        ind, dist = h.kneighbors(Q[good], 1)
        assert (ind >= 0).all() and not (dist > 1e-3).any()
        want = h.kneighbors(Q[good], 6)
    h.close()
