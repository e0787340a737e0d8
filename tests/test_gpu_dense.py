"""GPU: dense linkage in one thread-block cluster, bit for bit against the same
merge rules on the host: the closest pair by (distance, slot), Lance-Williams
updates in double rounded to float32, the merged cluster in the lower slot, a
cached nearest slot kept unless its cluster merged and got farther. Sizes around
the cluster's splits (1, 2, 4, 8 blocks), long rows, ties everywhere, duplicates,
negative cosine distances; and the form that spreads a merge over the whole GPU."""

import numpy as np
import pytest

import cuhc_b200 as C
from _data import blobs, grid, normal
from cuhc_b200 import _lib
from cuhc_b200._linkage import _dense_with_options

pytestmark = pytest.mark.gpu


def update(method, ak, bk, ab, na, nb, nk):
    if method == "single":
        return np.minimum(ak, bk)
    if method == "complete":
        return np.maximum(ak, bk)
    if method == "average":
        return (na * ak + nb * bk) / (na + nb)
    t = na + nb + nk
    return np.sqrt(np.maximum(((na + nk) * ak * ak + (nb + nk) * bk * bk - nk * ab * ab) / t, 0))


def merge_all(dist, method):
    """scipy-format tree of a float32 distance matrix."""
    n = len(dist)
    dist = dist.copy()
    np.fill_diagonal(dist, np.inf)
    size, ids, live = np.ones(n), np.arange(n), np.ones(n, bool)
    near = dist.argmin(1)
    gap = dist[np.arange(n), near]
    Z = np.empty((n - 1, 4))
    for step in range(n - 1):
        closest = int(gap.argmin())
        a, b = sorted((closest, int(near[closest])))
        ab = gap[closest]
        Z[step] = min(ids[a], ids[b]), max(ids[a], ids[b]), ab, size[a] + size[b]
        live[b], gap[b] = False, np.inf
        k = np.flatnonzero(live & (np.arange(n) != a))
        new = update(method, dist[a, k].astype(float), dist[b, k].astype(float), float(ab),
                     size[a], size[b], size[k]).astype(np.float32)
        dist[a, k] = dist[k, a] = new
        dist[b] = dist[:, b] = np.inf
        had = (near[k] == a) | (near[k] == b)
        take = np.where(had, new <= gap[k], new < gap[k])
        gap[k[take]], near[k[take]] = new[take], a
        for row in [*k[had & ~take], a]:
            near[row] = dist[row].argmin()
            gap[row] = dist[row, near[row]]
        size[a] += size[b]
        ids[a] = n + step
    return Z


CASES = {
    "2": lambda: normal(2, 3, seed=1),
    "3": lambda: normal(3, 3, seed=2),
    "128": lambda: blobs(128, 5, seed=3),
    "129": lambda: blobs(129, 5, seed=4),
    "257": lambda: normal(257, 16, seed=5),
    "513": lambda: blobs(513, 7, seed=6),
    "1100": lambda: normal(1100, 2, seed=7),
    "ties": lambda: grid(20),
    "duplicates": lambda: np.repeat(normal(40, 3, seed=8), 6, axis=0),
}


@pytest.mark.parametrize("method, metric", [("single", "euclidean"), ("complete", "manhattan"),
                                            ("average", "cosine"), ("ward", "euclidean")])
@pytest.mark.parametrize("name", CASES)
def test_merges_bit_for_bit(name, method, metric):
    X = CASES[name]()
    dist = C.pairwise_distances(X, metric=metric)
    got = C.linkage(X, method, metric=metric, algorithm="dense")
    np.testing.assert_array_equal(got, merge_all(dist, method))


@pytest.mark.parametrize("method, metric", [("single", "euclidean"), ("complete", "manhattan"),
                                            ("average", "cosine"), ("ward", "euclidean")])
@pytest.mark.parametrize("name", CASES)
def test_wide_merges_bit_for_bit(name, method, metric):
    """The form for many slots, at every size."""
    X = CASES[name]()
    dist = C.pairwise_distances(X, metric=metric)
    got = _dense_with_options(X, method, metric, resident_slots=0)
    np.testing.assert_array_equal(got, merge_all(dist, method))


@pytest.mark.parametrize("n, d", [(7168, 2), (7169, 2), (5120, 65), (5121, 65), (3072, 129),
                                  (3073, 129)])
def test_forms_agree_around_their_line(n, d):
    X = np.round(normal(n, d, seed=n) * 300).astype(np.float32)  # ties among long rows
    got = C.linkage(X, "complete")
    for slots in (0, n):
        np.testing.assert_array_equal(_dense_with_options(X, "complete", resident_slots=slots), got)


@pytest.mark.parametrize("slots", [0, 300])
def test_non_finite_distances_end_either_form(slots):
    X = normal(300, 4, seed=10)
    X[7] = 3e38  # its squared differences overflow: no finite distance
    tree = np.empty((299, 4))
    assert _lib.lib.cuhc_linkage_dense_with_options(
        _lib.float_ptr(X), 300, 4, 0, 2.0, 1, slots, _lib.double_ptr(tree)) < 0


def test_long_rows():
    X = normal(8300, 3, seed=9)
    single = C.linkage(X, "single", algorithm="dense")
    np.testing.assert_array_equal(single[:, 2], C.linkage(X, "single")[:, 2])


def test_non_finite_distances_are_refused():
    torch = pytest.importorskip("torch")
    X = torch.from_numpy(normal(300, 4, seed=10)).cuda()
    X[7] = float("nan")
    with pytest.raises(RuntimeError, match="NaN"):
        C.linkage(X, "complete")
