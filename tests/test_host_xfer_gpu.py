"""Large copies between pageable host memory and the device (the pinned ring):
the same results as small pieces give, over sizes at the ring's borders, both
storage orders, padded rows, host arrays with their own row pitch, from two
threads at once."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def warm(gpu, ab):
    """Enough traffic for the ring to be set up."""
    X = np.zeros((40_000, 512), np.float32)
    for _ in range(3):
        ab.KNN("s", order=0, algorithm="brute").fit(X).close()


@pytest.mark.parametrize("m,n,d", [(1023, 513, 8), (2048, 1024, 4), (3001, 1700, 37),
                                   (1, 600_000, 3), (700_001, 1, 5)])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("prec", ["s", "d"])
def test_pairwise_large_output(warm, ab, m, n, d, order, prec):
    """Blocks of 2 MB and more against the same distances in strips below that."""
    rng = np.random.default_rng(m + n)
    dt = np.float32 if prec == "s" else np.float64
    X, Y = rng.standard_normal((m, d)).astype(dt), rng.standard_normal((n, d)).astype(dt)
    st, D = ab.pairwise_distances(X, Y, "manhattan", prec=prec, order=order)
    assert st == 0
    strip = max(1, 100_000 // min(m, n))
    for a in range(0, max(m, n), strip * 7):  # every seventh strip
        sl = slice(a, a + strip)
        x, y = (X[sl], Y) if m >= n else (X, Y[sl])
        st, E = ab.pairwise_distances(x, y, "manhattan", prec=prec, order=order)
        np.testing.assert_array_equal(D[sl] if m >= n else D[:, sl], E)


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("n,d,pad", [(70_000, 37, 0), (60_000, 13, 9), (9_000, 300, 1)])
def test_upload_with_row_pitch(warm, ab, order, n, d, pad):
    """Training rows inside a wider array (leading dimension over the width)."""
    rng = np.random.default_rng(n)
    rows, cols = (n, d) if order == 0 else (d, n)
    big = rng.standard_normal((rows, cols + pad)).astype(np.float32)
    X = big[:, :cols] if order == 0 else big[:, :cols].T
    Q = np.ascontiguousarray(X[:50]) if order == 0 else np.asfortranarray(X[:50])
    res = []
    for dense in (False, True):
        nn = ab.KNN("s", order=order, metric="manhattan", algorithm="brute")
        if dense:
            nn.fit(np.array(X))
        else:
            nn.X = big
            nn.call("da_nn_set_data_s", n, d, big.ctypes.data_as(C.c_void_p), cols + pad)
        res.append(nn.kneighbors(Q, 3))
        nn.close()
    np.testing.assert_array_equal(res[0][0], res[1][0])
    np.testing.assert_array_equal(res[0][1], res[1][1])
    np.testing.assert_array_equal(res[0][0][:, 0], np.arange(50))


def test_two_threads(warm, ab):
    """Copies of two threads at once: one has the ring, the other goes without."""
    rng = np.random.default_rng(3)
    sets = [rng.standard_normal((60_000 + i, 24)).astype(np.float32) for i in range(2)]
    want, got = [None] * 2, [[], []]

    def fit(i):
        km = ab.KMeans(8, "s", order=0, n_init=1, max_iter=4)
        km.fit(sets[i], sets[i][:8])
        r = km.centres(8, 24), km.labels(len(sets[i])), km.transform(sets[i], 8)
        km.close()
        return r

    for i in range(2):
        want[i] = fit(i)

    def work(i):
        for _ in range(6):
            got[i].append(fit(i))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for i in range(2):
        assert len(got[i]) == 6
        for r in got[i]:
            for a, b in zip(r, want[i]):
                np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec", ["s", "d"])
def test_neighbours_many_results(warm, ab, prec):
    """Results over and under the size that comes back in one copy agree, in both
    orders."""
    rng = np.random.default_rng(5)
    dt = np.float32 if prec == "s" else np.float64
    X, Q = rng.standard_normal((4000, 9)).astype(dt), rng.standard_normal((9000, 9)).astype(dt)
    for order in (0, 1):
        nn = ab.KNN(prec, order=order, algorithm="brute").fit(X)
        ind, dist = nn.kneighbors(Q, 40)
        for a in (0, 4321, 8990):
            i, d = nn.kneighbors(Q[a:a + 10], 40)
            np.testing.assert_array_equal(ind[a:a + 10], i)
            np.testing.assert_array_equal(dist[a:a + 10], d)


@pytest.mark.parametrize("n,d", [(120_000, 40), (50_000, 150)])
def test_stream_set_after_the_data(warm, ab, n, d):
    """A stream that the handle is bound to after set_data reads all of the data
    (here the last rows hold each column's largest value), however much of the
    upload is still on its way."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(d)
    X = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    X[-d:] = np.diag(np.arange(2, d + 2, dtype=np.float32))
    streams = [torch.cuda.Stream() for _ in range(3)]
    for i in range(24):
        km = ab.KMeans(8, "s", order=ab.ROW_MAJOR, n_init=1, max_iter=1)
        km.set_data(X)
        km.L.da_b200_set_stream(km.h, C.c_void_p(streams[i % 3].cuda_stream))
        out = np.zeros(d, np.float32)
        km.call("da_b200_kmeans_shard_colmax_s", ab.ptr(out))
        km.close()
        np.testing.assert_array_equal(out, np.arange(2, d + 2, dtype=np.float32))


@pytest.mark.parametrize("order,d", [(0, 32), (0, 37), (1, 37)])
def test_page_locked_rows(warm, ab, order, d):
    """Page-locked training rows and outputs: the same results."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(d)
    n, m = 60_000, 900
    shape = (n, d) if order == 0 else (d, n)
    lock = torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()
    lock[:] = rng.standard_normal(shape)
    X = lock if order == 0 else lock.T
    Q = np.array(X[:m], order="C" if order == 0 else "F")
    res = []
    for rows in (X, np.array(X, order="C" if order == 0 else "F")):
        nn = ab.KNN("s", order=order, metric="manhattan", algorithm="brute").fit(rows)
        res.append(nn.kneighbors(Q, 3))
        nn.close()
        st, D = ab.pairwise_distances(rows[:m], rows[m:3 * m], "manhattan", prec="s", order=order)
        assert st == 0
        res[-1] += (D,)
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)
