"""One row whose width is no multiple of four features, uploaded into memory that
held something else: its pad on the device is zero, so that the searches that
read whole padded rows give what the same row gives among others."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def soil():
    """0xFF (NaN, -1) in free device memory.  The driver hands out small pieces of
    its blocks again as they were left, as long as something else holds the block."""
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    rt = C.CDLL("libcudart.so.12")  # torch's
    held = []
    for size in (64, 512, 4096, 65536):
        got = []
        for _ in range(256):
            p = C.c_void_p()
            assert rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0
            assert rt.cudaMemset(p, 0xFF, C.c_size_t(size)) == 0
            got.append(p)
        assert rt.cudaDeviceSynchronize() == 0
        held += got[1::2]
        for p in got[::2]:
            assert rt.cudaFree(p) == 0
    return lambda: [rt.cudaFree(p) for p in held]


@pytest.mark.parametrize("prec,d", [("s", 5), ("s", 37), ("d", 3)])
def test_one_query_of_an_ivf_index(gpu, ab, prec, d):
    dt = np.float32 if prec == "s" else np.float64
    rng = np.random.default_rng(d)
    X = rng.standard_normal((4000, d)).astype(dt)
    Q = rng.standard_normal((40, d)).astype(dt)

    def search(q):
        h = ab.ApproxNN(prec, order=ab.ROW_MAJOR, n_list=8, n_probe=3, seed=1)
        h.set_training_data(X).train_and_add()
        done = soil()
        r = h.kneighbors(q, 5)
        h.close()
        done()
        return r

    ind, dist = search(Q)
    for i in (0, 17, 39):
        one_ind, one_dist = search(Q[i:i + 1])
        np.testing.assert_array_equal(one_ind[0], ind[i])
        np.testing.assert_array_equal(one_dist[0], dist[i])


@pytest.mark.parametrize("d", [5, 13, 31])
def test_one_centre_of_a_batched_fit(gpu, ab, d):
    rng = np.random.default_rng(d)
    Xs = [rng.standard_normal((n, d)).astype(np.float32) for n in (1500, 1, 900)]
    Cs = [x[:1].copy() for x in Xs]
    for _ in range(3):
        done = soil()
        fits = ab.kmeans_batched(Xs, Cs, max_iter=20, tol=1e-4)
        done()
        for r, x in zip(fits, Xs):
            np.testing.assert_allclose(r["centres"][0], x.mean(0), atol=1e-5)
            assert not np.asarray(r["labels"]).any()
            ss = ((x - x.astype(np.float64).mean(0)) ** 2).sum()
            np.testing.assert_allclose(r["inertia"], ss, rtol=1e-5, atol=1e-9)
