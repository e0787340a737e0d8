"""Performance cases of cuhc_b200: the calls that a program using it makes, over the sizes,
dimensions, metrics and options that its configurations, tests and benchmark use.

A case is a plain dict:
  op        "hdbscan" (the HDBSCAN estimator), "linkage" (a merge tree), "batch" (many small
            trees in one call), "pairwise" (a distance matrix)
  data      "blobs" (Gaussian blobs + uniform noise), "normal" (standard normal) or
            "aniso" (Gaussian blobs with their own covariances + uniform noise)
  on        "host" (NumPy arrays, as a scikit-learn program passes them) or "gpu" (a CUDA tensor)
"""

import math

import numpy as np
import torch

import cuhc_b200 as cuhc


def listed():
    return [
        # The smallest calls: a few hundred points (the size of most test sets), where a call is
        # launches, copies and host work.
        dict(name="hdbscan-400x8", op="hdbscan", data="blobs", on="host", n=400, d=8,
             min_cluster_size=5, metric="euclidean"),
        dict(name="single-1000x2", op="linkage", data="blobs", on="host", n=1000, d=2,
             method="single", metric="euclidean"),
        # The plain single-linkage configuration, 20,000 x 32 standard normal.
        dict(name="single-20000x32", op="linkage", data="normal", on="host", n=20_000, d=32,
             method="single", metric="euclidean"),
        # An ordinary density clustering of 100,000 points, arrays on the host.
        dict(name="hdbscan-100000x8", op="hdbscan", data="blobs", on="host", n=100_000, d=8,
             min_cluster_size=25, metric="euclidean"),
        # The headline clustering: 1,000,000 x 8, 20 blobs and 10 % noise, min_samples 25, whole
        # estimator (tree, core distances, labels, probabilities), points already on the GPU.
        dict(name="hdbscan-1000000x8", op="hdbscan", data="blobs", on="gpu", n=1_000_000, d=8,
             min_cluster_size=25, metric="euclidean"),
        # More than 32 features (embeddings after a projection) and an odd count.
        dict(name="hdbscan-50001x50", op="hdbscan", data="blobs", on="gpu", n=50_001, d=50,
             min_cluster_size=15, metric="euclidean"),
        # Single linkage where no box separates anything: standard normal in 32 dimensions.
        dict(name="single-300000x32", op="linkage", data="normal", on="gpu", n=300_000, d=32,
             method="single", metric="euclidean"),
        # Single linkage of 50 anisotropic clusters in 16 dimensions.
        dict(name="single-500000x16", op="linkage", data="aniso", on="gpu", n=500_000, d=16,
             method="single", metric="euclidean"),
        # Ward's tree of 200,000 x 32 standard normal points.
        dict(name="ward-200000x32", op="linkage", data="normal", on="gpu", n=200_000, d=32,
             method="ward", metric="euclidean"),
        # Many uneven problems at once: 256 instances, n log-uniform in [64, 50,000], 2, 8 or 32
        # features, alternately single linkage and HDBSCAN's tree with min_samples 10.
        dict(name="batch-256", op="batch", data="blobs", on="host", count=256, low=64, high=50_000,
             min_samples=10, metric="euclidean"),
        # A linkage that needs the full matrix, at an odd size.
        dict(name="average-3001x16", op="linkage", data="blobs", on="host", n=3001, d=16,
             method="average", metric="euclidean"),
        # A distance matrix that stays on the GPU (1 GiB).
        dict(name="pairwise-16384x64", op="pairwise", data="normal", on="gpu", n=16_384, m=16_384,
             d=64, metric="euclidean"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(["hdbscan", "hdbscan", "single", "single", "ward", "dense", "batch",
                     "pairwise"])
    on = rng.choice(["host", "gpu"])
    if op == "hdbscan":
        metric = rng.choice(["euclidean", "euclidean", "euclidean", "manhattan", "cosine"])
        d = rng.choice([2, 3, 5, 8, 11, 16, 24, 32, 50, 64])
        high = 1_000_000 if d <= 8 else 300_000 if d <= 16 else 50_000
        n = _log_int(rng, 400, min(high, 60_000) if metric != "euclidean" else high)
        return dict(op="hdbscan", data=rng.choice(["blobs", "blobs", "aniso"]), on=on, n=n, d=d,
                    min_cluster_size=_log_int(rng, 5, 60), metric=metric)
    if op == "single":
        metric = rng.choice(["euclidean", "euclidean", "euclidean", "sqeuclidean", "chebyshev",
                             "cosine"])
        d = rng.choice([2, 4, 7, 8, 13, 16, 31, 32, 48])
        high = 500_000 if d <= 16 else 300_000 if d <= 32 else 60_000
        n = _log_int(rng, 1000, min(high, 60_000) if metric in ("chebyshev", "cosine") else high)
        data = rng.choice(["blobs", "aniso"] if n > 100_000 else ["blobs", "normal", "aniso"])
        return dict(op="linkage", data=data, on=on, n=n, d=d, method="single", metric=metric)
    if op == "ward":
        return dict(op="linkage", data=rng.choice(["blobs", "normal"]), on=on,
                    n=_log_int(rng, 1000, 200_000), d=rng.choice([2, 5, 8, 16, 27, 32]),
                    method="ward", metric="euclidean")
    if op == "dense":
        return dict(op="linkage", data="blobs", on=on, n=_log_int(rng, 300, 3000),
                    d=rng.choice([2, 7, 16, 40]), method=rng.choice(["complete", "average"]),
                    metric=rng.choice(["euclidean", "manhattan", "cosine"]))
    if op == "batch":
        return dict(op="batch", data="blobs", on="host", count=_log_int(rng, 16, 256), low=64,
                    high=_log_int(rng, 1000, 50_000), min_samples=rng.choice([5, 10, 16]),
                    metric="euclidean")
    return dict(op="pairwise", data="normal", on=on, n=_log_int(rng, 200, 16_384 if on == "gpu"
                                                                else 4000),
                m=_log_int(rng, 200, 16_384 if on == "gpu" else 4000),
                d=rng.choice([3, 8, 17, 32, 64, 100]),
                metric=rng.choice(["euclidean", "sqeuclidean", "manhattan", "chebyshev", "cosine"]))


# ---------------------------------------------------------------------------
# Data


def _points(kind, n, d, rng):
    """n x d float32 points on the GPU, drawn from the torch.Generator rng."""
    def normal(*shape):
        return torch.randn(*shape, generator=rng, device="cuda")

    def uniform(*shape):
        return torch.rand(*shape, generator=rng, device="cuda")

    if kind == "normal":
        return normal(n, d)
    count = 20 if kind == "blobs" else 50
    noise = n // 10 if kind == "blobs" else n // 20
    label = torch.randint(count, (n - noise,), generator=rng, device="cuda")
    centres = uniform(count, d) * 20 - 10
    if kind == "blobs":
        inside = centres[label] + normal(n - noise, d)
    else:
        # Every cluster its own covariance: eigenvalues log-uniform in [0.05, 5].
        scale = torch.exp(uniform(count, d) * math.log(100.0)) * 0.05
        basis = torch.linalg.qr(normal(count, d, d))[0]
        inside = normal(n - noise, d)
        for c in range(count):
            rows = label == c
            inside[rows] = centres[c] + (inside[rows] * scale[c].sqrt()) @ basis[c]
    low, high = inside.min(0).values, inside.max(0).values
    points = torch.cat([inside, low + (high - low) * uniform(noise, d)])
    return points[torch.randperm(n, generator=rng, device="cuda")].contiguous()


def _instances(case, seed):
    """The batch's problems: 1-12 blobs of standard deviation 0.5-2 and 5 % noise each. Sizes
    and dimensions belong to the case, the points to the seed."""
    shape, rng = np.random.default_rng(case["count"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(shape.uniform(math.log(case["low"]), math.log(case["high"])))))
        d, blobs = int(shape.choice([2, 8, 32])), int(rng.integers(1, 13))
        noise = int(round(0.05 * n))
        label = rng.integers(0, blobs, n - noise)
        centres, stds = rng.uniform(-10, 10, (blobs, d)), rng.uniform(0.5, 2.0, blobs)
        inside = centres[label] + rng.standard_normal((n - noise, d)) * stds[label, None]
        points = np.vstack([inside, rng.uniform(inside.min(0), inside.max(0), (noise, d))])
        out.append(np.ascontiguousarray(points[rng.permutation(n)], dtype=np.float32))
    return out


def _ranks(case):
    return [case["min_samples"] if i % 2 else 0 for i in range(case["count"])]


def _inputs(case, seed):
    rng = torch.Generator(device="cuda")
    rng.manual_seed(seed)
    arrays = [_points(case["data"], case["n"], case["d"], rng)]
    if case["op"] == "pairwise":
        arrays.append(_points(case["data"], case["m"], case["d"], rng))
    return arrays


def prepare(case, seed):
    if case["op"] == "batch":
        return dict(case=case, X=_instances(case, seed), min_samples=_ranks(case))
    arrays = _inputs(case, seed)
    if case["on"] == "host":
        arrays = [a.cpu().numpy() for a in arrays]
    return dict(case=case, X=arrays[0], Y=arrays[-1])


def run(state):
    case, X = state["case"], state["X"]
    if case["op"] == "hdbscan":
        model = cuhc.HDBSCAN(min_cluster_size=case["min_cluster_size"],
                             metric=case["metric"]).fit(X)
        tree = model._single_linkage_tree_
        return dict(labels=model.labels_, probabilities=model.probabilities_,
                    core=model.core_distances_, tree=tree, heights=tree[:, 2])
    if case["op"] == "linkage":
        tree = cuhc.linkage(X, case["method"], metric=case["metric"])
        return dict(tree=tree, heights=tree[:, 2])
    if case["op"] == "batch":
        trees, cores = zip(*cuhc.batched_trees(X, state["min_samples"], metric=case["metric"]))
        return dict(trees=np.concatenate(trees), core=np.concatenate(cores))
    return cuhc.pairwise_distances(X, state["Y"], metric=case["metric"])


# ---------------------------------------------------------------------------
# Work, tolerance and the 64-bit answers


def work(case):
    """Bytes: the points once, the results once. Operations: 3 per feature and pair that has to be
    looked at: every pair of a distance matrix (half of a symmetric one), and every pair of
    standard normal points (no bound excludes any); for clustered data the neighbours that the
    answer names (min_samples a point, one for a merge tree)."""
    if case["op"] == "batch":
        # Log-uniform sizes: mean (high - low) / ln(high / low) points, 14 features on average.
        n = case["count"] * (case["high"] - case["low"]) / math.log(case["high"] / case["low"])
        pairs = n * (1 + case["min_samples"] / 2)
        return {"bytes": n * (4 * 14 + 32 + 4), "flops": 3 * 14 * pairs}
    n, d = case["n"], case["d"]
    if case["op"] == "pairwise":
        return {"bytes": 4 * ((n + case["m"]) * d + n * case["m"]), "flops": 3 * d * n * case["m"]}
    if case["op"] == "hdbscan":
        out, pairs = 32 + 4 + 8 + 8, n * case["min_cluster_size"]
    else:
        every = case["data"] == "normal" or case["method"] in ("complete", "average")
        out, pairs = 32, n * (n - 1) / 2 if every else n
    return {"bytes": n * (4 * d + out), "flops": 3 * d * pairs}


def tolerance(case):
    if case["op"] == "pairwise":
        # 32-bit sums of up to 100 features.
        return {"rel": 2e-6}
    # Trees, core distances and labels are exact in every mode of the library: the same 32-bit
    # distances, ties by point index.
    return "exact"


def _distances(A, B, metric):
    """len(A) x len(B) float64 distances of float64 tensors, feature by feature."""
    if metric == "cosine":
        def unit(x):
            return x / x.norm(dim=1, keepdim=True).clamp_min(1e-300)
        return 1 - unit(A) @ unit(B).T
    out = torch.zeros(len(A), len(B), dtype=torch.float64, device=A.device)
    for f in range(A.shape[1]):
        gap = A[:, f, None] - B[None, :, f]
        if metric in ("euclidean", "sqeuclidean"):
            out.addcmul_(gap, gap)
        elif metric == "manhattan":
            out.add_(gap.abs_())
        else:
            torch.maximum(out, gap.abs_(), out=out)
    return out.sqrt_() if metric == "euclidean" else out


def _core(X, k, metric):
    """The k-th smallest distance of every row, the row itself counted as 0."""
    n = len(X)
    rows = max(1, (1 << 26) // n)
    out = []
    for first in range(0, n, rows):
        dist = _distances(X[first:first + rows], X, metric)
        at = torch.arange(len(dist), device=X.device)
        dist[at, first + at] = 0
        out.append(dist.topk(k, largest=False).values.max(1).values)
    return torch.cat(out)


def _spanning_heights(dist):
    """Sorted edge weights of the minimum spanning tree of a full matrix (Prim)."""
    n = len(dist)
    best = dist[0].clone()
    outside = torch.zeros(n, dtype=torch.float64, device=dist.device)
    outside[0] = math.inf
    heights = torch.empty(n - 1, dtype=torch.float64, device=dist.device)
    for i in range(n - 1):
        weight, at = torch.min(best + outside, 0)
        heights[i] = weight
        outside[at] = math.inf
        best = torch.minimum(best, dist[at])
    return heights.sort().values


def _dense_heights(dist, method):
    """Merge heights of complete or average linkage (the closest pair each time)."""
    n = len(dist)
    np.fill_diagonal(dist, np.inf)
    size = np.ones(n)
    near = dist.argmin(1)
    gap = dist[np.arange(n), near]
    heights = []
    for _ in range(n - 1):
        a = int(gap.argmin())
        b = int(near[a])
        heights.append(gap[a])
        merged = (np.maximum(dist[a], dist[b]) if method == "complete" else
                  (size[a] * dist[a] + size[b] * dist[b]) / (size[a] + size[b]))
        merged[[a, b]] = np.inf
        size[a] += size[b]
        dist[a], dist[:, a] = merged, merged
        dist[b], dist[:, b] = np.inf, np.inf
        gap[b] = np.inf
        closer = merged < gap
        gap[closer], near[closer] = merged[closer], a
        for row in np.flatnonzero(((near == a) | (near == b)) & ~closer & np.isfinite(gap)):
            near[row] = dist[row].argmin()
            gap[row] = dist[row, near[row]]
        near[a] = merged.argmin()
        gap[a] = merged[near[a]]
    return np.array(heights)


def exact(case, seed):
    if case["op"] == "batch":
        out = []
        for X, k in zip(_instances(case, seed), _ranks(case)):
            X = torch.from_numpy(X).cuda().double()
            out.append(_core(X, k, case["metric"]).cpu().numpy() if k else np.zeros(len(X)))
        return dict(trees=None, core=np.concatenate(out))
    arrays = [a.double() for a in _inputs(case, seed)]
    if case["op"] == "pairwise":
        out = _distances(*arrays, case["metric"])
        return out if case["on"] == "gpu" else out.cpu().numpy()
    X, n = arrays[0], case["n"]
    if case["op"] == "hdbscan":
        if n > 100_000:
            return None
        core = _core(X, case["min_cluster_size"], case["metric"])
        heights = None
        if n <= 20_000:
            reach = torch.maximum(_distances(X, X, case["metric"]),
                                  torch.maximum(core[:, None], core[None, :]))
            heights = _spanning_heights(reach).cpu().numpy()
        return dict(labels=None, probabilities=None, core=core.cpu().numpy(), tree=None,
                    heights=heights)
    if n > 20_000 or case["method"] == "ward":
        return None
    dist = _distances(X, X, case["metric"])
    heights = (_spanning_heights(dist).cpu().numpy() if case["method"] == "single" else
               _dense_heights(dist.cpu().numpy(), case["method"]))
    return dict(tree=None, heights=heights)
