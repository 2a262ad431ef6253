"""A handle's first search takes its lists in batches of a megabyte where a few are
enough, later ones in one: the same neighbours, and the oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def launches(nn):
    ms, n = C.c_double(), C.c_int32()
    assert nn.L.da_b200_get_kernel_time(nn.h, b"knn_select", C.byref(ms), C.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("prec,n,nq,k,metric", [("s", 3000, 500, 40, "euclidean"),
                                                ("d", 900, 500, 10, "cosine"),
                                                ("d", 5000, 190, 5, "manhattan")])
@pytest.mark.parametrize("order", [0, 1])
def test_batches(gpu, ab, orc, prec, n, nq, k, metric, order):
    rng = np.random.default_rng(n)
    dt = np.float32 if prec == "s" else np.float64
    X, Q = rng.standard_normal((n, 13)).astype(dt), rng.standard_normal((nq, 13)).astype(dt)
    nn = ab.KNN(prec, order=order, metric=metric, algorithm="brute").fit(X)
    nn.L.da_b200_set_kernel_timing(nn.h, 1)
    first = nn.kneighbors(Q, k)
    batches = launches(nn)
    second = nn.kneighbors(Q, k)
    assert 2 <= batches <= 4 and launches(nn) == batches + 1
    oi, od = orc.knn(X, Q, k, metric)
    for ind, dist in (first, second):
        np.testing.assert_array_equal(ind, oi)
        np.testing.assert_array_equal(dist, od)
    nn.close()


@pytest.mark.parametrize("n,k", [(1, 1), (17, 16), (200, 1), (300, 30), (2047, 100), (1100, 120)])
@pytest.mark.parametrize("kind", ["random", "sorted", "equal"])
def test_lists_of_small_sets(gpu, ab, orc, n, k, kind):
    """All rows are sampled: short lists, also where the neighbours lie together."""
    rng = np.random.default_rng(n + k)
    X = rng.standard_normal((n, 5))
    if kind == "sorted":
        X = X[np.argsort(X[:, 0])] * [50, 1, 1, 1, 1]
    elif kind == "equal":
        X[:] = X[0]
    Q = X[rng.integers(0, n, 60)] + 0.1
    for prec, dt in (("s", np.float32), ("d", np.float64)):
        nn = ab.KNN(prec, metric="euclidean", algorithm="brute").fit(X.astype(dt))
        ind, dist = nn.kneighbors(Q.astype(dt), k)
        oi, od = orc.knn(X.astype(dt), Q.astype(dt), k, "euclidean")
        np.testing.assert_array_equal(ind, oi)
        np.testing.assert_array_equal(dist, od)
        nn.close()
