"""Radius searches that the tensor-core path refuses (more than one pair in eight a
candidate): the next ones go past it, ever longer, and smaller radii take it; its
statistic stands for the whole search."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def launches(nn, name):
    ms, n = C.c_double(), C.c_int32()
    assert nn.L.da_b200_get_kernel_time(nn.h, name, C.byref(ms), C.byref(n)) == 0
    return n.value


def test_refused_searches(gpu, ab):
    rng = np.random.default_rng(0)
    X = rng.standard_normal((40_000, 32)).astype(np.float32)
    Q = rng.standard_normal((4_000, 32)).astype(np.float32)
    nn = ab.KNN("s", order=0, algorithm="brute").fit(X)
    nn.radius_neighbors(Q, 1.0, True, False)
    assert nn.stat("tensor_core") == 1
    nn.L.da_b200_set_kernel_timing(nn.h, 1)
    few = Q[:400]
    for _ in range(12):
        dense = nn.radius_neighbors(few, 9.0, True, False)
        assert nn.stat("tensor_core") == 0
    # one block of distances a search, and a mask at the 1st, 3rd, 6th and 11th
    assert launches(nn, b"radius_distances") == 12 + 4
    sparse = nn.radius_neighbors(few, 4.0, True, False)
    assert nn.stat("tensor_core") == 1
    nn.set("precision mode", "plain")
    for got, radius in ((dense, 9.0), (sparse, 4.0)):
        for a, b in zip(got, nn.radius_neighbors(few, radius, True, False)):
            np.testing.assert_array_equal(a, b)
    nn.close()


def test_blocks_of_both_kinds(gpu, ab):
    """The first block of queries has no neighbours, the last one is dense."""
    rng = np.random.default_rng(1)
    n, d = 400_000, 8
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[:100_000] *= np.float32(0.01)
    Q = 50 + rng.standard_normal((5_400, d)).astype(np.float32)  # blocks of 5,248 and 152
    Q[-100:] = 0
    nn = ab.KNN("s", order=0, algorithm="brute").fit(X)
    cnt, off, ind, dist = nn.radius_neighbors(Q, 0.5, True, False)
    assert nn.stat("tensor_core") == 0
    assert not cnt[:5_300].any() and (cnt[5_300:5_400] >= 100_000).all()
    nn.set("precision mode", "plain")
    for a, b in zip((cnt, off, ind, dist), nn.radius_neighbors(Q, 0.5, True, False)):
        np.testing.assert_array_equal(a, b)
    nn.close()
