"""The radius search's tensor-core path (fp32 euclidean): counts, rows and
distances equal to the plain path's and the oracle's, bit for bit, at the edges
of its tiles (128 queries, 256 rows, 64 features), with rows on the radius
itself, without any hit, in an order of values where the bf16 products say
little, and where a block goes to the plain path (no finite threshold, too many
candidates)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stat(nn):
    v = C.c_double()
    nn.L.da_b200_get_stat(nn.h, b"tensor_core", C.byref(v))
    return v.value


def both(ab, X, Q, radius, sort=False, order=0, metric="euclidean"):
    """(tensor-core path taken, its result, the plain path's)."""
    nn = ab.KNN("s", order=order, metric=metric, algorithm="brute").fit(X)
    for _ in range(9):  # a handle's first small searches are plain
        got = nn.radius_neighbors(Q, radius, True, sort)
        if stat(nn):
            break
    taken = stat(nn)
    nn.set("precision mode", "plain")
    want = nn.radius_neighbors(Q, radius, True, sort)
    assert stat(nn) == 0
    nn.close()
    return taken, got, want


@pytest.mark.parametrize("n,nq,d", [(16384, 500, 64), (16385, 129, 257), (40_001, 128, 100),
                                    (70_000, 1, 128), (65_537, 127, 65), (300_000, 257, 7),
                                    (100_255, 600, 33), (32_769, 129, 127)])
@pytest.mark.parametrize("order,sort,metric", [(0, False, "euclidean"), (1, True, "sqeuclidean")])
def test_radius_tc_equals_plain(gpu, ab, orc, n, nq, d, order, sort, metric):
    rng = np.random.default_rng(n + nq)
    means = rng.uniform(-4, 4, (50, d))
    X = (means[rng.integers(0, 50, n)] + rng.standard_normal((n, d))).astype(np.float32)
    Q = (means[rng.integers(0, 50, nq)] + rng.standard_normal((nq, d))).astype(np.float32)
    if d % 2 == 0:  # whole numbers: many rows exactly on the radius
        X, Q = np.round(X), np.round(Q)
    Q[0] = X[n - 1]
    # a distance that occurs, so that the test at the radius is one of equality
    e = np.linalg.norm(X[:20_000].astype(np.float64) - Q[0].astype(np.float64), axis=1)
    r = np.float32(np.sort(e)[60])
    radius = float(r * r if metric == "sqeuclidean" else r)
    if order:
        X, Q = np.asfortranarray(X), np.asfortranarray(Q)
    taken, got, want = both(ab, X, Q, radius, sort, order, metric)
    assert taken == (d <= 128)  # wider rows do not fit the kernel's shared memory
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    for q, (ri, rd) in enumerate(orc.radius(X, Q[:2], radius, metric, 2.0, sort)):
        assert got[0][q] == len(ri)
        np.testing.assert_array_equal(got[2][got[1][q]:][:len(ri)], ri)
        np.testing.assert_array_equal(got[3][got[1][q]:][:len(ri)], rd.astype(np.float32))


@pytest.mark.parametrize("form,taken", [("none", 1), ("far", None), ("infinite", 0), ("dense", 0),
                                        ("nan row", 1), ("crowded", 1)])
def test_radius_tc_forms(gpu, ab, form, taken):
    rng = np.random.default_rng(len(form))
    X = rng.standard_normal((50_000, 32)).astype(np.float32)
    Q = rng.standard_normal((400, 32)).astype(np.float32)
    radius = {"none": 0.01, "dense": 9.0}.get(form, 4.5)
    if form == "far":        # |x|^2 is 3e5 times the squared distances
        X, Q = X + 3000, Q + 3000
    elif form == "infinite":
        Q[7, 3] = np.inf
    elif form == "nan row":  # within no radius of any query
        X[11, 4] = np.nan
    elif form == "crowded":  # a query with more rows than the kernel's list
        X[10_000:14_000] = X[9_999]
        Q[3] = X[9_999]
    got_tc, got, want = both(ab, X, Q, radius)
    if taken is not None:
        assert got_tc == taken
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
