"""A handle bound to a stream, given its data, then bound to another: what follows
on the second stream sees the data, whatever the first one still had to do."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def warm(gpu, ab):
    """Enough traffic for the transfer ring: uploads of a few MB then return with
    the copies queued."""
    X = np.zeros((40_000, 512), np.float32)
    for _ in range(3):
        ab.KNN("s", order=0, algorithm="brute").fit(X).close()


def bind(ab, h, stream):
    assert h.L.da_b200_set_stream(h.h, C.c_void_p(stream)) == 0


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("to", ["stream", "own", "per thread"])
def test_from_stream_to_stream(warm, ab, order, to):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(order)
    n, d = 30_000, 40
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    second = {"stream": b.cuda_stream, "own": None, "per thread": 2}[to]
    for rep in range(3):
        X = rng.uniform(-1, 1, (n, d)).astype(np.float32)
        X[-d:] = np.diag(np.arange(2, d + 2, dtype=np.float32))
        X = X if order == 0 else np.asfortranarray(X)
        km = ab.KMeans(8, "s", order=order, n_init=1, max_iter=1)
        bind(ab, km, a.cuda_stream)
        with torch.cuda.stream(a):
            torch.cuda._sleep(20_000_000)  # about 10 ms
        km.set_data(X)
        bind(ab, km, second)
        out = np.zeros(d, np.float32)
        km.call("da_b200_kmeans_shard_colmax_s", ab.ptr(out))
        km.close()
        np.testing.assert_array_equal(out, np.arange(2, d + 2, dtype=np.float32))

        nn = ab.KNN("s", order=order, metric="manhattan", algorithm="brute")
        bind(ab, nn, a.cuda_stream)
        with torch.cuda.stream(a):
            torch.cuda._sleep(20_000_000)
        nn.fit(X)
        bind(ab, nn, second)
        Q = X[-64:] if order == 0 else np.asfortranarray(X[-64:])
        ind, dist = nn.kneighbors(Q, 1)
        nn.close()
        np.testing.assert_array_equal(ind[:, 0], np.arange(n - 64, n))
        assert not dist.any()


def test_first_stream_destroyed(warm, ab):
    """The first stream is gone by the time that the handle is bound again."""
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    rt = C.CDLL("libcudart.so.12")  # torch's
    X = np.random.default_rng(1).uniform(-1, 1, (30_000, 40)).astype(np.float32)
    for _ in range(3):
        s = C.c_void_p()
        assert rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
        nn = ab.KNN("s", order=0, metric="manhattan", algorithm="brute")
        bind(ab, nn, s.value)
        nn.fit(X)
        assert rt.cudaStreamDestroy(s) == 0
        bind(ab, nn, None)
        ind, _ = nn.kneighbors(X[-64:], 1)
        nn.close()
        np.testing.assert_array_equal(ind[:, 0], np.arange(len(X) - 64, len(X)))
