"""The tensor-core kNN pass at the sizes where its tiles, sample and lists change
shape, against the plain path on the same data (equal, bit for bit): one query
and one over a 128-query tile, a last row tile of one row, a last K block of
16 columns, the smallest set it takes with the largest k, more queries than one
batch of lists, rows sorted so that all neighbours lie in one work item."""
import numpy as np
import pytest

from test_knn_tc_gpu import mixture, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nq,d,k,metric,kind", [
    (65_537, 129, 64, 10, "euclidean", ""),
    (130_817, 128, 80, 100, "sqeuclidean", ""),
    (16_384, 500, 128, 256, "euclidean", ""),
    (20_000, 1_000, 33, 1, "cosine", ""),
    (70_000, 257, 128, 256, "cosine", ""),
    (40_000, 16_500, 32, 5, "euclidean", ""),
    (200_000, 64, 64, 50, "euclidean", "sorted"),
    (100_000, 130, 100, 33, "euclidean", "shifted"),
])
def test_knn_tc_sizes(gpu, ab, nx, nq, d, k, metric, kind):
    rng = np.random.default_rng(nx + nq)
    X = mixture(rng, nx, d, comps=40)
    if kind == "sorted":
        X = X[np.argsort(X[:, 0])]
    if kind == "shifted":  # margins of many times the distances' spread
        X += np.float32(60)
    Q = X[rng.integers(0, nx, nq)] + rng.standard_normal((nq, d)).astype(np.float32)
    pi, pd, ptc, _ = run(ab, X, Q, k, metric, "plain", nq % 2)
    ti, td, ttc, _ = run(ab, X, Q, k, metric, "bf16x3", nq % 2)
    assert ptc == 0.0 and ttc == 1.0
    np.testing.assert_array_equal(td, pd)
    np.testing.assert_array_equal(ti, pi)
