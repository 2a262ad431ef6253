"""Buffers that only make a call faster: where one of them is not to be had, the
call does without (each device allocation failed in turn, as in
test_alloc_failure_gpu.py) and gives the same results."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENV = "AOCLDA_B200_FAIL_ALLOC"


def sweep(ab, setup, call, needed):
    """Fail the call's first, second, ... allocation, each time on a fresh handle.
    `needed` of them are what the call cannot do without."""
    def run(n):
        h = setup()
        try:
            if n:
                os.environ[ENV] = str(n)
            return call(h)
        finally:
            os.environ.pop(ENV, None)
            if h is not None:
                h.close()

    want, refused = run(0), 0
    for n in range(1, 30):
        try:
            got = run(n)
        except ab.DAError as e:
            assert e.status == 2
            refused += 1
            continue
        for a, b in zip(got, want):
            np.testing.assert_array_equal(np.asarray(a), np.asarray(b))
    assert refused <= needed, refused


def knn(ab, n, d, nq, k, prec="s", order=0, metric="euclidean", cyclic=0, fit_fails=False):
    rng = np.random.default_rng(n + d)
    dt = np.float32 if prec == "s" else np.float64
    X, Q = rng.standard_normal((n, d)).astype(dt), rng.standard_normal((nq, d)).astype(dt)
    if cyclic:
        c = rng.uniform(-5, 5, (cyclic, d))
        X += c[np.arange(n) % cyclic].astype(dt)
        Q += c[rng.integers(0, cyclic, nq)].astype(dt)

    def make():
        h = ab.KNN(prec, order=order, metric=metric, algorithm="brute")
        return h if fit_fails else h.fit(X)

    def call(h):
        if fit_fails:
            h.fit(X)
        return h.kneighbors(Q, k)

    return make, call


# queries; queries' norms, rows' norms, results
@pytest.mark.parametrize("metric,needed", [("euclidean", 2), ("cosine", 4)])
@pytest.mark.parametrize("n,d,nq,cyclic", [(20_000, 64, 500, 0), (70_000, 96, 300, 19),
                                           (3_000, 16, 700, 0)])
def test_neighbours(gpu, ab, metric, needed, n, d, nq, cyclic):
    sweep(ab, *knn(ab, n, d, nq, 10, metric=metric, cyclic=cyclic), needed)


@pytest.mark.parametrize("prec,order", [("s", 0), ("d", 0)])
def test_rows_padded_on_the_device(gpu, ab, prec, order):
    """Dense rows of a width that the device pads: rows, queries, results."""
    sweep(ab, *knn(ab, 5_000, 37, 200, 5, prec, order, "manhattan", fit_fails=True), 3)


def test_transposed_results(gpu, ab):
    """Column-major: the uploads' transposing needs its stage (one for both)."""
    sweep(ab, *knn(ab, 4_000, 12, 9_000, 30, "d", 1), 3)


@pytest.mark.parametrize("ties", [0, 6000])
def test_queries_searched_again(gpu, ab, ties):
    rng = np.random.default_rng(1)
    X = rng.standard_normal((30_000, 20)).astype(np.float32)
    X[:ties] = X[0]
    Q = np.vstack([X[:5], rng.standard_normal((500, 20)).astype(np.float32)])
    # queries, results, the running lists' two
    sweep(ab, lambda: ab.KNN("s", order=0, metric="manhattan", algorithm="brute").fit(X),
          lambda h: h.kneighbors(Q, 5), 4)


def test_radius(gpu, ab):
    rng = np.random.default_rng(2)
    X = rng.standard_normal((40_000, 32)).astype(np.float32)
    Q = rng.standard_normal((2_000, 32)).astype(np.float32)

    # queries, distances, counts, offsets, hits, rows, values
    sweep(ab, lambda: ab.KNN("s", order=0, algorithm="brute").fit(X), lambda h: h.radius_neighbors(Q, 4.5, True, False), 7)


@pytest.mark.parametrize("d", [36, 37])
def test_pairwise(gpu, ab, d):
    rng = np.random.default_rng(d)
    X, Y = rng.standard_normal((700, d)), rng.standard_normal((300, d))

    def call(_):
        st, D = ab.pairwise_distances(X, Y, metric="euclidean", prec="d", order=0)
        if st != 0:
            raise ab.DAError(st, "da_pairwise_distances_d")
        return (D,)

    sweep(ab, lambda: None, call, 5)
