"""fp64 Lloyd fits one after another on a handle: the first iterations are the
host's, then the loop's graph takes over, within a fit, in the next ones and after
a change of the data; results as from the host loop alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def blobs(seed, n, d, k):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, d)) + 2.0 * rng.integers(0, 3, (n, 1))
    return X, X[rng.choice(n, k, replace=False)].copy()


def fit(km, X, C0):
    km.fit(X, C0)
    return km.labels(len(X)), km.centres(*C0.shape), km.rinfo(), km.stat("graph_loop")


def test_fits_on_one_handle(gpu, ab):
    sets = [blobs(0, 4000, 9, 6), blobs(1, 3000, 9, 6), blobs(2, 4000, 9, 6)]

    def run(host):
        km = ab.KMeans(6, "d", order=ab.ROW_MAJOR, max_iter=40, n_init=1)
        km.set("convergence tolerance", 0.0)
        km.L.da_b200_set_kernel_timing(km.h, host)
        out = [fit(km, *sets[i]) for i in (0, 0, 1, 1, 2, 2, 0)]
        km.close()
        return out

    host, got = run(1), run(0)
    assert [r[3] for r in host] == [0.0] * 7
    taken = [r[3] for r in got]
    iters = [int(r[2][3]) for r in got]
    assert iters[0] > 14 and taken[0] == 1 and taken[1] == 1, (iters, taken)
    for h, g in zip(host, got):
        for a, b in zip(h[:3], g[:3]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("max_iter", [1, 2, 3])
def test_short_fits(gpu, ab, max_iter):
    """Fits too short for a graph of their own; after some of them it is there."""
    X, C0 = blobs(3, 2500, 7, 5)
    km = ab.KMeans(5, "d", order=ab.ROW_MAJOR, max_iter=max_iter, n_init=1)
    km.set("convergence tolerance", 0.0)
    got = [fit(km, X, C0) for _ in range(20)]
    km.close()
    assert got[0][3] == 0
    assert got[-1][3] == (1.0 if max_iter > 1 else 0.0)
    for r in got[1:]:
        for a, b in zip(r[:3], got[0][:3]):
            np.testing.assert_array_equal(a, b)
