"""Performance cases of the distance, nearest-neighbour and k-means entry points.

Every pass goes through the public binding with host arrays, as the C API takes
them: the upload of that call's inputs and the download of its results belong to
it.  What a program keeps between calls (a handle holding its training data or
its fitted model) is made in prepare().

Data are isotropic Gaussian mixtures (means U[-5, 5]^d, sigma 1), the recipe of
the repository's benchmark, generated on the GPU from the seed and copied to
host arrays in the case's storage order.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..",
                                "aocl-data-analytics_b200"))
import aoclda_b200 as ab  # noqa: E402

LARGEST_FLOPS = 1.0e12  # of a drawn case; the largest listed ones are at or above it


def listed():
    return [
        # a few rows against a few rows in the API's defaults (fp64, column-major):
        # the smallest call, all latency
        dict(name="pairwise_small_f64", kind="pairwise", prec="d", order="col", m=64, n=50, d=20,
             metric="euclidean"),
        # a kernel-matrix / clustering preprocessing block: odd sizes, the output dominates
        dict(name="pairwise_block_f32", kind="pairwise", prec="s", order="row", m=4001, n=3001,
             d=96, metric="euclidean"),
        # fp64 neighbours and classification of a test set (the repository's plain kNN workload)
        dict(name="knn_classify_f64", kind="classify", prec="d", order="col", n=10_000, nq=2_000,
             d=32, k=10, comps=16, weights="uniform"),
        # one interactive query against a resident index
        dict(name="knn_one_query_f32", kind="knn", prec="s", order="row", n=1_000_000, nq=1, d=96,
             k=10, comps=512, metric="euclidean"),
        # a mid-sized table with a city-block metric and a ragged width
        dict(name="knn_manhattan_f32", kind="knn", prec="s", order="row", n=50_000, nq=1_000, d=37,
             k=5, comps=64, metric="manhattan"),
        # batch neighbours of a large embedding table, the largest kNN call
        dict(name="knn_batch_f32", kind="knn", prec="s", order="row", n=1_000_000, nq=4_096, d=128,
             k=100, comps=1024, metric="euclidean"),
        # radius neighbours (DBSCAN-like use), results read back through the result queries
        dict(name="radius_f32", kind="radius", prec="s", order="row", n=200_000, nq=2_000, d=32,
             comps=256, reach=0.85),
        # the headline k-means fit: k-means++ and up to 50 Lloyd iterations, data uploaded
        dict(name="kmeans_fit_f32", kind="kmeans", prec="s", order="row", n=1_000_000, d=64, k=256,
             comps=256, init="k-means++", max_iter=50),
        # an fp64 fit from centres that the caller has, default storage order
        dict(name="kmeans_fit_f64", kind="kmeans", prec="d", order="col", n=100_000, d=20, k=16,
             comps=24, init="supplied", max_iter=30),
        # labels and distances of new rows under a fitted model
        dict(name="kmeans_apply_f32", kind="apply", prec="s", order="row", n=20_000, m=100_000,
             d=32, k=64, comps=64),
        # approximate search over inverted lists
        dict(name="ivf_search_f32", kind="ivf", prec="s", order="row", n=200_000, nq=5_000, d=96,
             k=10, comps=512, n_list=512, n_probe=16),
        # many small fits at once: per-customer / per-segment clusterings of uneven sizes
        dict(name="kmeans_many_f32", kind="many", sets=48, n=20_000, max_iter=30),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pairwise", "pairwise", "knn", "knn", "knn", "knn", "classify", "radius",
                       "kmeans", "kmeans", "apply", "ivf", "many"])
    prec, order = rng.choice("ssd"), rng.choice(["row", "col"])
    if kind == "pairwise":
        return dict(kind=kind, prec=prec, order=order, m=_log(rng, 10, 4000),
                    n=_log(rng, 10, 4000), d=_log(rng, 2, 200),
                    metric=rng.choice(["euclidean", "euclidean", "sqeuclidean", "manhattan",
                                       "cosine"]))
    if kind == "knn":
        metric = rng.choice(["euclidean", "euclidean", "euclidean", "sqeuclidean", "cosine",
                             "manhattan", "inner product"])
        d, k = _log(rng, 4, 128), rng.choice([1, 5, 10, 30, 100])
        n, nq = _log(rng, 1000, 1_000_000), _log(rng, 1, 4096)
        most = LARGEST_FLOPS if prec == "s" else LARGEST_FLOPS / 16
        nq = max(1, min(nq, int(most / (2.0 * n * d))))
        return dict(kind=kind, prec=prec, order=order, n=n, nq=nq, d=d, k=k,
                    comps=max(4, n // 1000), metric=metric)
    if kind == "classify":
        return dict(kind=kind, prec=prec, order=order, n=_log(rng, 500, 50_000),
                    nq=_log(rng, 1, 4000), d=_log(rng, 4, 64), k=rng.randint(1, 20),
                    comps=rng.randint(2, 24), weights=rng.choice(["uniform", "distance"]))
    if kind == "radius":
        n = _log(rng, 2000, 400_000)
        return dict(kind=kind, prec=prec, order=order, n=n, nq=_log(rng, 1, 2000),
                    d=_log(rng, 8, 64), comps=max(4, n // 800), reach=rng.uniform(0.8, 0.9))
    if kind == "kmeans":
        n = _log(rng, 2000, 1_000_000 if prec == "s" else 200_000)
        k = min(_log(rng, 4, 256 if prec == "s" else 64), n // 20)
        return dict(kind=kind, prec=prec, order=order, n=n, d=_log(rng, 4, 64), k=k, comps=k,
                    init=rng.choice(["k-means++", "supplied"]), max_iter=rng.randint(10, 50))
    if kind == "apply":
        k = _log(rng, 4, 256)
        return dict(kind=kind, prec=prec, order=order, n=max(4000, 40 * k),
                    m=_log(rng, 1, 100_000), d=_log(rng, 4, 128), k=k, comps=k)
    if kind == "ivf":
        n = _log(rng, 20_000, 200_000)
        return dict(kind=kind, prec=prec, order=order, n=n, nq=_log(rng, 1, 5000),
                    d=_log(rng, 8, 128), k=rng.choice([1, 10, 50]), comps=max(16, n // 400),
                    n_list=rng.choice([64, 256, 512]), n_probe=rng.choice([4, 8, 16]))
    return dict(kind="many", sets=rng.randint(4, 64), n=_log(rng, 3000, 20_000),
                max_iter=rng.randint(5, 30))


# ------------------------------------------------------------------ inputs --
class _Data:
    """Draws of one mixture: generator, component means."""

    def __init__(self, seed, d, comps):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.means = torch.rand(comps, d, generator=self.g, device="cuda") * 10 - 5

    def rows(self, n):
        lab = torch.randint(len(self.means), (n,), generator=self.g, device="cuda")
        x = torch.randn(n, self.means.shape[1], generator=self.g, device="cuda")
        return x.add_(self.means[lab]), lab


def _dtype(case):
    return torch.float64 if case.get("prec") == "d" else torch.float32


def _order(case):
    return ab.ROW_MAJOR if case["order"] == "row" else ab.COLUMN_MAJOR


def _host(case, x):
    """A host array of the case's type and storage order."""
    x = x.to(_dtype(case))
    return x.cpu().numpy() if case["order"] == "row" else x.t().contiguous().cpu().numpy().T


def _radius(case):
    # two rows of one component lie sqrt(2 d) apart on average
    return case["reach"] * math.sqrt(2.0 * case["d"])


def _radius_room(case):
    # a component has about 800 rows, at most two fifths of them within reach
    return 600 * case["nq"] + 1000


def _many_shapes(case, seed):
    """Rows, features, clusters of every data set: uneven, as segments are."""
    r = np.random.RandomState(seed)
    n = np.clip(np.exp(r.normal(math.log(case["n"]), 1.0, case["sets"])), 1000, 200_000)
    total = 1.5 * case["sets"] * case["n"]
    n = np.maximum(1000, n * min(1.0, total / n.sum())).astype(int)
    return [(int(a), int(r.choice([16, 32, 64])), int(r.randint(8, 65))) for a in n]


def _inputs(case, seed):
    """The case's inputs as GPU tensors."""
    kind = case["kind"]
    if kind == "many":
        sets = []
        for i, (n, d, k) in enumerate(_many_shapes(case, 7)):
            x, _ = _Data(seed * 1000 + i, d, k).rows(n)
            sets.append((x, x[:k].clone()))
        return dict(sets=sets)
    comps = case.get("comps", 8)
    data = _Data(seed, case["d"], comps)
    if kind == "pairwise":
        return dict(x=data.rows(case["m"])[0], y=data.rows(case["n"])[0])
    x, lab = data.rows(case["n"])
    out = dict(x=x, lab=lab)
    if kind in ("knn", "classify", "radius", "ivf"):
        out["q"] = data.rows(case["nq"])[0]
    if kind == "apply":
        out["q"] = data.rows(case["m"])[0]
    if kind in ("kmeans", "apply"):
        out["c0"] = x[torch.randperm(case["n"], generator=data.g, device="cuda")[:case["k"]]]
    return out


def prepare(case, seed):
    t = _inputs(case, seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "many":
        s["x"] = [x.cpu().numpy() for x, _ in t["sets"]]
        s["c0"] = [c.cpu().numpy() for _, c in t["sets"]]
        return s
    s.update({k: _host(case, v) for k, v in t.items() if k != "lab"})
    prec, order = case["prec"], _order(case)
    if kind == "knn":
        s["h"] = ab.KNN(prec, order=order, metric=case["metric"], algorithm="brute").fit(s["x"])
    elif kind == "classify":
        s["h"] = ab.KNN(prec, order=order, number_of_neighbors=case["k"], weights=case["weights"],
                        algorithm="brute").fit(s["x"], t["lab"].cpu().numpy().astype(np.int32))
    elif kind == "radius":
        s["h"] = ab.KNN(prec, order=order, algorithm="brute").fit(s["x"])
        # the program's result tables, large enough for any of its queries
        s["ind"] = np.zeros(_radius_room(case), np.int32)
        s["dist"] = np.zeros(_radius_room(case), s["x"].dtype)
    elif kind == "kmeans":
        s["h"] = ab.KMeans(case["k"], prec, order=order, n_init=1, seed=1,
                           max_iter=case["max_iter"], initialization_method=case["init"])
    elif kind == "apply":
        s["h"] = ab.KMeans(case["k"], prec, order=order, n_init=1, max_iter=5).fit(s["x"], s["c0"])
    elif kind == "ivf":
        s["h"] = ab.ApproxNN(prec, order=order, n_list=case["n_list"], n_probe=case["n_probe"],
                             kmeans_iter=8, seed=1).set_training_data(s["x"]).train_and_add()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "pairwise":
        return ab.pairwise_distances(s["x"], s["y"], metric=case["metric"], prec=case["prec"],
                                     order=_order(case))[1]
    if kind in ("knn", "ivf"):
        ind, dist = s["h"].kneighbors(s["q"], case["k"])
        return {"indices": ind, "distances": dist}
    if kind == "classify":
        ind, dist = s["h"].kneighbors(s["q"], case["k"])
        return {"indices": ind, "distances": dist, "labels": s["h"].predict(s["q"])}
    if kind == "radius":
        cnt, off, ind, dist = s["h"].radius_neighbors(s["q"], _radius(case))
        s["ind"][:len(ind)] = ind
        s["dist"][:len(dist)] = dist
        return {"count": cnt, "offsets": off, "indices": s["ind"], "distances": s["dist"]}
    if kind == "kmeans":
        h = s["h"].fit(s["x"], s["c0"] if case["init"] == "supplied" else None)
        info = h.rinfo()
        return {"centres": h.centres(case["k"], case["d"]), "labels": h.labels(case["n"]),
                "iterations": int(info[3]), "inertia": info[4]}
    if kind == "apply":
        return {"labels": s["h"].predict(s["q"]),
                "distances": s["h"].transform(s["q"], case["k"])}
    fits = ab.kmeans_batched(s["x"], s["c0"], max_iter=case["max_iter"])
    return {"centres": np.concatenate([f["centres"].ravel() for f in fits]),
            "labels": np.concatenate([f["labels"] for f in fits]),
            "iterations": np.array([f["n_iter"] for f in fits]),
            "inertia": np.array([f["inertia"] for f in fits])}


def work(case):
    """What a pass cannot do without: inputs read once, results written once, the
    multiply-adds of the distances (three operations per feature where the
    differences are squared or summed as they are)."""
    e = 8 if case.get("prec") == "d" else 4
    kind, d = case["kind"], case.get("d", 0)
    if kind == "pairwise":
        m, n = case["m"], case["n"]
        per = 2 if case["metric"] == "cosine" else 3
        return {"bytes": e * ((m + n) * d + m * n), "flops": per * m * n * d}
    if kind in ("knn", "classify"):
        n, nq, k = case["n"], case["nq"], case["k"]
        per = 3 if case.get("metric") == "manhattan" else 2
        calls = 2 if kind == "classify" else 1
        return {"bytes": calls * (e * (n + nq) * d + nq * k * (e + 4)),
                "flops": calls * per * n * nq * d}
    if kind == "radius":
        n, nq = case["n"], case["nq"]
        return {"bytes": e * (n + nq) * d + nq * 60 * (e + 4), "flops": 2 * n * nq * d}
    if kind == "kmeans":
        n, k = case["n"], case["k"]
        trials = 2 + int(math.log(k)) if case["init"] == "k-means++" else 0
        its = case["max_iter"]
        return {"bytes": e * n * d * (1 + its + (k if trials else 0)) + 4 * n,
                "flops": 2 * n * d * k * (its + trials)}
    if kind == "apply":
        m, k = case["m"], case["k"]
        return {"bytes": e * m * (2 * d + k) + 4 * m, "flops": 4 * m * d * k}
    if kind == "ivf":
        n, nq = case["n"], case["nq"]
        rows = n * case["n_probe"] / case["n_list"]
        return {"bytes": e * (n + nq) * d + nq * case["k"] * (e + 4),
                "flops": 2 * nq * d * (rows + case["n_list"])}
    shapes = _many_shapes(case, 7)
    its = case["max_iter"]
    return {"bytes": sum(4 * n * d * (1 + its) for n, d, _ in shapes),
            "flops": sum(2 * n * d * k * its for n, d, k in shapes)}


# ------------------------------------------------------- 64-bit references --
def _distances(metric, x, y):
    """Distances of the rows of x (..., 1, d) to the rows of y (..., r, d), fp64."""
    if metric == "cosine":
        return 1 - (x * y).sum(-1) / (x.norm(dim=-1) * y.norm(dim=-1))
    if metric == "inner product":
        return (x * y).sum(-1)
    if metric == "manhattan":
        return (x - y).abs().sum(-1)
    sq = (x - y).square().sum(-1)
    return sq if metric == "sqeuclidean" else sq.sqrt()


def _neighbours(metric, x, q, k):
    """Distances of the k nearest rows: a pass over all rows finds a few more than k
    candidates, whose distances are then taken directly."""
    best = []
    step = max(1, int(4e9 / (8 * len(x))))
    if metric == "manhattan":
        step = max(1, int(4e9 / (8 * len(x) * x.shape[1])))
    sq = x.square().sum(1)
    for a in range(0, len(q), step):
        b = q[a:a + step]
        if metric == "manhattan":
            score = torch.cdist(b, x, p=1)
        elif metric == "cosine":
            score = -(b @ x.t()) / sq.sqrt()
        elif metric == "inner product":
            score = -(b @ x.t())
        else:
            score = sq - 2 * (b @ x.t())
        near = score.topk(min(len(x), k + 8), largest=False).indices
        dist = _distances(metric, b[:, None], x[near])
        best.append(dist.topk(k, largest=metric == "inner product").values)
    return torch.cat(best)


def _lloyd(x, c, max_iter, tol=1e-4):
    """Lloyd's iterations as the entry points do them: (centres, labels, iterations)."""
    def nearest(c):
        cn = c.square().sum(1)
        step = max(1, int(2e9 / (8 * len(c))))
        return torch.cat([(cn - 2 * (b @ c.t())).argmin(1) for b in x.split(step)])

    prev, n_iter, relabel = None, max_iter, True
    for it in range(max_iter):
        lab = nearest(c)
        old = c
        cnt = torch.bincount(lab, minlength=len(c))
        c = torch.zeros_like(c).index_add_(0, lab, x) / cnt.clamp(min=1)[:, None]
        if it > 1 and torch.equal(lab, prev):
            n_iter, relabel = it, False
            break
        if (c - old).norm() < tol * old.norm():
            n_iter = it
            break
        prev = lab
    return c, nearest(c) if relabel else lab, n_iter


def _inertia(x, c, lab):
    return (x - c[lab]).square().sum().cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "ivf" or (kind == "kmeans" and case["init"] == "k-means++"):
        return None  # depend on the trained lists, on the drawn centres
    t = _inputs(case, seed)
    if kind == "many":
        cs, inertia = [], []
        for x, c0 in t["sets"]:
            x = x.double()
            c, lab, _ = _lloyd(x, c0.double(), case["max_iter"])
            cs.append(c.ravel())
            inertia.append(_inertia(x, c, lab))
        return {"centres": torch.cat(cs).cpu(), "labels": None, "iterations": None,
                "inertia": torch.stack(inertia)}
    t = {k: v.to(_dtype(case)).double() if k != "lab" else v for k, v in t.items()}
    if kind == "pairwise":
        step = max(1, int(2e9 / (8 * case["n"] * case["d"])))
        return torch.cat([_distances(case["metric"], b[:, None], t["y"])
                          for b in t["x"].split(step)]).cpu()
    if kind in ("knn", "classify"):
        dist = _neighbours(case.get("metric", "euclidean"), t["x"], t["q"], case["k"])
        return {"indices": None, "distances": dist.cpu(), "labels": None}
    if kind == "radius":
        out = []
        for b in t["q"].split(max(1, int(2e9 / (8 * case["n"] * case["d"])))):
            dist = _distances("euclidean", b[:, None], t["x"])
            out.append(dist[dist <= _radius(case)])
        dist = torch.zeros(_radius_room(case), dtype=torch.float64)
        found = torch.cat(out).cpu()
        dist[:len(found)] = found
        return {"count": None, "offsets": None, "indices": None, "distances": dist}
    if kind == "kmeans":
        c, lab, _ = _lloyd(t["x"], t["c0"], case["max_iter"])
        return {"centres": c.cpu(), "labels": None, "iterations": None,
                "inertia": _inertia(t["x"], c, lab)}
    c, _, _ = _lloyd(t["x"], t["c0"], 5)
    sq = t["q"].square().sum(1)[:, None] - 2 * (t["q"] @ c.t()) + c.square().sum(1)
    return {"labels": None, "distances": sq.clamp(min=0).sqrt().cpu()}
