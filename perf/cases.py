"""Performance cases of flashlib_b200: what its users have it do, through the public entry points.

A case is a dict of plain values.  ``listed()`` gives the named ones, ``draw(rng)`` one more of the same
ranges, ``prepare`` what a program holds before the call (fitted estimators, indexes, query batches),
``run`` one call, ``work`` the bytes and operations that call cannot do without, ``tolerance`` how far
another correct implementation's results may lie.

Kinds of work:

``knn``        ``NearestNeighbors.fit`` once, ``kneighbors`` per batch of queries: from one query of an
               interactive lookup to the batches of an offline join; fp32, bf16 and fp16 rows.
``knn_batch``  ``flash_knn`` on ``(B, N, D)``: many small independent problems (point clouds, feature sets).
``kmeans``     ``flash_kmeans`` with given start centroids and a fixed number of iterations; ``batch`` > 1
               trains that many independent codebooks in one call.
``kmeans_fit`` ``KMeans.fit`` with its defaults: random start, convergence test every iteration.
``predict``    ``KMeans.predict``: labels of rows under fitted centroids.
``ivf``        ``IVFFlat.fit`` once, ``kneighbors`` per batch of queries.
"""
import torch

import flashlib_b200 as fl

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one query against a resident database: the lookup behind an interactive request
        dict(name="knn_online", kind="knn", nq=1, m=1_000_000, d=128, k=10, dtype="fp32", data="mixture"),
        # the repository's small configuration: 20 000 rows, 1 000 queries
        dict(name="knn_small", kind="knn", nq=1_000, m=20_000, d=64, k=10, dtype="fp32", data="randn"),
        # the benchmark configuration: 10 000 queries against 1 000 000 x 128 non-negative rows
        dict(name="knn_bulk", kind="knn", nq=10_000, m=1_000_000, d=128, k=10, dtype="fp32", data="mixture"),
        # one GPU's share of the 100 000 000-row configuration: many neighbours, the largest call
        dict(name="knn_shard_k100", kind="knn", nq=100_000, m=12_500_000, d=96, k=100, dtype="fp32", data="randn"),
        # unit-length embedding rows stored in 16 bits, more features than one operand tile holds
        dict(name="knn_embed_bf16", kind="knn", nq=2_000, m=200_000, d=768, k=10, dtype="bf16", data="unit"),
        # neighbourhoods within point clouds: 32 clouds of 2 048 points, three coordinates
        dict(name="knn_clouds", kind="knn_batch", batch=32, nq=2_048, m=2_048, d=3, k=16),
        # the k-means configuration: 1 000 000 x 128, 1 024 clusters, 20 Lloyd iterations
        dict(name="kmeans_1m", kind="kmeans", batch=1, n=1_000_000, d=128, K=1024, iters=20),
        # a set of product-quantiser codebooks: 16 sub-spaces of 8 features, 256 centroids each
        dict(name="kmeans_codebooks", kind="kmeans", batch=16, n=65_536, d=8, K=256, iters=10),
        # an ordinary small clustering with the estimator's defaults, ragged sizes
        dict(name="kmeans_fit_small", kind="kmeans_fit", n=50_001, d=33, K=50, iters=25),
        # labels of a quarter million rows under 500 fitted centroids, ragged sizes
        dict(name="kmeans_predict", kind="predict", n=250_001, d=96, K=500),
        # the inverted-file configuration: 1 024 lists, 16 probed, 10 000 queries
        dict(name="ivf_bulk", kind="ivf", nq=10_000, m=1_000_000, d=128, nlist=1024, nprobe=16, k=10),
        # the same index under a trickle of queries
        dict(name="ivf_online", kind="ivf", nq=16, m=1_000_000, d=128, nlist=1024, nprobe=16, k=10),
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def _features(rng, lo, hi):
    """A feature count: as often a multiple of 8, as real rows mostly are, as any number."""
    d = _log(rng, lo, hi)
    return max(8, d // 8 * 8) if rng.random() < 0.7 else d


def draw(rng):
    kind = rng.choice(["knn", "knn", "knn", "embed", "knn_batch", "kmeans", "kmeans_fit", "predict", "ivf", "ivf"])
    if kind == "knn":
        return dict(kind="knn", nq=_log(rng, 1, 20_000), m=_log(rng, 10_000, 2_000_000), d=_features(rng, 16, 256),
                    k=_log(rng, 1, 100), dtype="fp32", data=rng.choice(["mixture", "randn"]))
    if kind == "embed":
        return dict(kind="knn", nq=_log(rng, 1, 4_000), m=_log(rng, 20_000, 400_000), d=_features(rng, 256, 1024),
                    k=_log(rng, 1, 50), dtype=rng.choice(["bf16", "fp16"]), data="unit")
    if kind == "knn_batch":
        n = _log(rng, 128, 4_000)
        return dict(kind="knn_batch", batch=_log(rng, 2, 64), nq=n, m=n, d=rng.choice([2, 3, 3, 6, 16, 64]), k=_log(rng, 1, 40))
    if kind == "kmeans":
        if rng.random() < 0.5:
            return dict(kind="kmeans", batch=_log(rng, 4, 32), n=_log(rng, 4_000, 100_000), d=rng.choice([4, 8, 8, 16]),
                        K=rng.choice([16, 64, 256]), iters=rng.randint(3, 20))
        return dict(kind="kmeans", batch=1, n=_log(rng, 50_000, 1_500_000), d=_features(rng, 32, 256), K=_log(rng, 64, 2048),
                    iters=rng.randint(3, 20))
    if kind == "kmeans_fit":
        return dict(kind="kmeans_fit", n=_log(rng, 2_000, 200_000), d=_features(rng, 8, 128), K=_log(rng, 8, 200), iters=25)
    if kind == "predict":
        return dict(kind="predict", n=_log(rng, 1_000, 1_000_000), d=_features(rng, 16, 256), K=_log(rng, 10, 2_000))
    m = _log(rng, 50_000, 1_000_000)
    nlist = _log(rng, 64, 1024)
    return dict(kind="ivf", nq=_log(rng, 1, 20_000), m=m, d=_features(rng, 32, 256), nlist=nlist, nprobe=min(nlist, _log(rng, 4, 48)),
                k=_log(rng, 1, 50))


def _rows(data, n, d, g, means=None):
    """``n`` rows on the GPU: ``randn`` N(0, 1); ``mixture`` a Gaussian mixture clamped at zero
    (non-negative descriptors); ``blobs`` the same without the clamp; ``unit`` unit-length embeddings
    scattered around common directions."""
    x = torch.randn(n, d, generator=g, device="cuda")
    if data != "randn":
        step = 1 << 20
        for s in range(0, n, step):
            part = x[s:s + step]
            comp = torch.randint(0, means.shape[0], (part.shape[0],), generator=g, device="cuda")
            part.add_(means[comp])
        if data == "mixture":
            x.clamp_min_(0.0)
        elif data == "unit":
            x.div_(x.norm(dim=1, keepdim=True))
    return x


def _means(data, n_comp, d, g):
    if data == "randn":
        return None
    return (1.0 if data == "unit" else 2.0) * torch.randn(n_comp, d, generator=g, device="cuda")


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = dict(case)
    kind = c["kind"]
    state = {"kind": kind}
    if kind == "knn":
        dt = DTYPES[c["dtype"]]
        means = _means(c["data"], max(16, c["m"] // 244), c["d"], g)
        db = _rows(c["data"], c["m"], c["d"], g, means).to(dt)
        state["q"] = _rows(c["data"], c["nq"], c["d"], g, means).to(dt)
        state["nn"] = fl.NearestNeighbors(n_neighbors=c["k"]).fit(db)
    elif kind == "knn_batch":
        state["x"] = torch.randn(c["batch"], c["nq"], c["d"], generator=g, device="cuda")
        state["k"] = c["k"]
    elif kind == "kmeans":
        b, n, d, K = c["batch"], c["n"], c["d"], c["K"]
        x = torch.stack([_rows("blobs", n, d, g, _means("blobs", K, d, g)) for _ in range(b)])
        state.update(x=x if b > 1 else x[0], K=K, iters=c["iters"])
        state["init"] = (x[:, :K] if b > 1 else x[0, :K]).clone()
    elif kind == "kmeans_fit":
        state["x"] = _rows("blobs", c["n"], c["d"], g, _means("blobs", c["K"], c["d"], g))
        state["km"] = fl.KMeans(c["d"], c["K"], niter=c["iters"])
    elif kind == "predict":
        means = _means("blobs", c["K"], c["d"], g)
        km = fl.KMeans(c["d"], c["K"], niter=3, tol=0.0)
        state["km"] = km.fit(_rows("blobs", max(20 * c["K"], 2_000), c["d"], g, means))
        state["x"] = _rows("blobs", c["n"], c["d"], g, means)
    elif kind == "ivf":
        means = _means("mixture", max(16, c["m"] // 244), c["d"], g)
        torch.manual_seed(seed)          # the index's k-means start is drawn from the global generator
        ivf = fl.IVFFlat(nlist=c["nlist"], nprobe=c["nprobe"], n_neighbors=c["k"], niter=10)
        state["ivf"] = ivf.fit(_rows("mixture", c["m"], c["d"], g, means))
        state["q"] = _rows("mixture", c["nq"], c["d"], g, means)
    return state


def run(state):
    kind = state["kind"]
    if kind == "knn":
        return state["nn"].kneighbors(state["q"])
    if kind == "knn_batch":
        return fl.flash_knn(state["x"], state["x"], state["k"])
    if kind == "kmeans":
        labels, centroids, _ = fl.flash_kmeans(state["x"], state["K"], max_iters=state["iters"], init_centroids=state["init"])
        return labels, centroids
    if kind == "kmeans_fit":
        km = state["km"].fit(state["x"])
        return km.cluster_ids_b, km.centroids_b
    if kind == "predict":
        return state["km"].predict(state["x"])
    return state["ivf"].kneighbors(state["q"])


def work(case):
    c = case
    kind = c["kind"]
    if kind == "knn":
        size = 4 if c["dtype"] == "fp32" else 2
        return {"bytes": (c["m"] + c["nq"]) * c["d"] * size + c["nq"] * c["k"] * 8, "flops": 2.0 * c["nq"] * c["m"] * c["d"]}
    if kind == "knn_batch":
        b = c["batch"]
        return {"bytes": b * (c["m"] * c["d"] * 4 + c["nq"] * c["k"] * 8), "flops": 2.0 * b * c["nq"] * c["m"] * c["d"]}
    if kind in ("kmeans", "kmeans_fit"):
        b = c.get("batch", 1)
        # an iteration needs the inner products of every row with every centroid and every row's sum
        # (kmeans_fit: `iters` is the most it runs; it ends when no centroid moves)
        return {"bytes": b * (c["n"] * c["d"] * 4 + 2 * c["K"] * c["d"] * 4 + c["n"] * 4),
                "flops": float(c["iters"]) * b * (2.0 * c["n"] * c["K"] * c["d"] + c["n"] * c["d"])}
    if kind == "predict":
        return {"bytes": (c["n"] + c["K"]) * c["d"] * 4 + c["n"] * 4, "flops": 2.0 * c["n"] * c["K"] * c["d"]}
    pairs = c["nq"] * c["nprobe"]
    rows = min(c["m"], pairs * c["m"] / c["nlist"])         # rows of the lists that are probed at all
    return {"bytes": (rows + c["nlist"] + c["nq"]) * c["d"] * 4 + c["nq"] * c["k"] * 12,
            "flops": 2.0 * c["nq"] * c["nlist"] * c["d"] + 2.0 * pairs * (c["m"] / c["nlist"]) * c["d"]}


def tolerance(case):
    kind = case["kind"]
    if kind in ("knn", "knn_batch"):
        # fp32 sums of squares; neighbours whose distances agree to the last bits may change places
        return {"rel": 1e-5, "max": 1e-3, "differ": 2e-3}
    if kind == "predict":
        # rows on the boundary between two centroids, whose sums are accumulated in no fixed order
        return {"rel": 1e-5, "differ": 1e-3}
    if kind in ("kmeans", "kmeans_fit"):
        # the sums have no fixed order: a row that changes sides moves two centroids by 1 / (rows of a
        # cluster), and the iterations after it carry that on (two runs of one build: rel 1e-3)
        return {"rel": 2e-3, "max": 0.2, "differ": 2e-3}
    # as knn, on an index trained by k-means: rows on list boundaries may sit in either list (two runs of
    # one build: rel 1.5e-3, 0.3 % of the neighbours)
    return {"rel": 3e-3, "max": 0.3, "differ": 6e-3}
