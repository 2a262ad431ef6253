"""Lloyd with the update by counting sort (fp64), few clusters and many: the
loop run as a graph against the same loop run from the host (kernel timing keeps
it there), bit for bit, and labels against a NumPy assignment with the final
centres; at the edges of the assignment's tiles (8, 16, 32 clusters, 128 rows, 32
features), of the sort's blocks (256 and 1,024 rows, 32 and 256 clusters) and
with clusters that stay empty."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fit(ab, X, C0, host, max_iter, tol):
    km = ab.KMeans(C0.shape[0], "d", order=ab.ROW_MAJOR, max_iter=max_iter, n_init=1)
    km.set("convergence tolerance", tol)
    km.L.da_b200_set_kernel_timing(km.h, int(host))
    km.fit(X, C0)
    v = C.c_double()
    km.L.da_b200_get_stat(km.h, b"graph_loop", C.byref(v))
    out = km.labels(X.shape[0]), km.centres(*C0.shape), km.rinfo(), km.predict(X[: len(X) // 2 + 1])
    km.close()
    return out, v.value


@pytest.mark.parametrize("n,d,k", [(129, 3, 1), (128, 32, 8), (1025, 33, 9), (70_000, 20, 17),
                                   (65_536, 31, 32), (20_000, 5, 32), (4097, 64, 33), (5000, 129, 16),
                                   (3000, 7, 256), (2049, 130, 257)])
@pytest.mark.parametrize("max_iter,tol,empty", [(12, 0.0, False), (40, 1e-3, True)])
def test_sort_loop(gpu, ab, n, d, k, max_iter, tol, empty):
    rng = np.random.default_rng(n + d + k)
    X = rng.standard_normal((n, d)) + rng.integers(0, 3, (n, 1)) * 4.0
    C0 = X[rng.choice(n, min(k, n), replace=False)].copy()
    if empty and k > 2:  # a copy never wins a tie; one far from every row
        C0[1], C0[2] = C0[0], 1e6
    host, graph = fit(ab, X, C0, True, max_iter, tol), fit(ab, X, C0, False, max_iter, tol)
    assert host[1] == 0
    for a, b in zip(host[0], graph[0]):
        np.testing.assert_array_equal(a, b)
    lab, cen = graph[0][0], graph[0][1]
    if int(graph[0][2][3]) == max_iter:  # relabelled against the final centres
        v = (cen * cen).sum(1)[None] - 2 * X @ cen.T
        best = v.min(1)
        own = v[np.arange(n), lab]
        # |x|^2 scale times the rounding of d + 2 products
        assert (own - best <= 4 * (d + 2) * 2.0 ** -53 * ((X * X).sum(1) + (cen * cen).sum(1).max())).all()
    np.testing.assert_array_equal(graph[0][3], lab[: n // 2 + 1])
