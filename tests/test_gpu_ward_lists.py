"""GPU: RNN-Ward with nearest neighbours kept across rounds.

Rounds search only the clusters whose kept list no longer proves their nearest
neighbour. The oracle searches every cluster against every other in every
round, in the same float32 arithmetic (its divisions are IEEE where the
selection uses the fast division, within 2 ulp: the data below has no weights
that close other than exact ties, which both resolve by index). Merges must be
identical; heights to float32 rounding of one division and square root (the
bound below: 4 units in the last place). Data: tile edges, several feature
chunks, far from the origin (where stored centroids are coarse against the
distances), exact ties, duplicates, clusters of very different sizes.
"""

import numpy as np
import pytest

from _data import blobs, grid, normal
from cuhc_b200 import _lib
from cuhc_b200._linkage import _ward_rnn_with_lists, _ward_rnn_with_options

pytestmark = pytest.mark.gpu
f4, f8 = np.float32, np.float64


def squared(a, b):
    """|a - b|^2 by fused multiply-adds in feature order (rows broadcast)."""
    acc = np.zeros(np.broadcast_shapes(a.shape[:-1], b.shape[:-1]), f4)
    for k in range(a.shape[-1]):
        gap = (a[..., k] - b[..., k]).astype(f8)
        acc = (gap * gap + acc.astype(f8)).astype(f4)
    return acc


def ward_rounds(X):
    """[(rep, rep, height)] of reciprocal-nearest-neighbour rounds."""
    cent, size, rep = X.astype(f4), np.ones(len(X), f4), np.arange(len(X))
    merges = []
    while len(rep) > 1:
        near = np.empty(len(rep), np.int64)
        for i in range(len(rep)):
            s = squared(cent[i], cent)
            w = f4(2) * (size[i] * size) * s / (size[i] + size)
            w[i] = np.inf
            near[i] = np.lexsort((rep, w))[0]
        pairs = [(i, j) for i, j in enumerate(near) if near[j] == i and rep[i] < rep[j]]
        assert pairs
        gone = []
        for i, j in pairs:
            h = f4(2) * (size[i] * size[j]) / (size[i] + size[j]) * squared(cent[i], cent[j])
            merges.append((rep[i], rep[j], np.sqrt(h)))
        for i, j in pairs:
            step = (size[j] / (size[i] + size[j])).astype(f8)
            cent[i] = ((cent[j] - cent[i]).astype(f8) * step + cent[i].astype(f8)).astype(f4)
            size[i] += size[j]
            gone.append(j)
        keep = np.setdiff1d(np.arange(len(rep)), gone)
        cent, size, rep = cent[keep], size[keep], rep[keep]
    return merges


def clusters(merges, n):
    """{(smallest point, size): height}, heights non-decreasing up the tree."""
    up, size, height, out = np.arange(n), np.ones(n, int), np.zeros(n, f4), {}
    for u, v, h in merges:  # a representative is its cluster's smallest point
        h = max(h, height[u], height[v])
        up[v], height[u] = u, h
        size[u] += size[v]
        out[(int(u), int(size[u]))] = h
    return out


def tree_clusters(Z):
    n = len(Z) + 1
    smallest = np.concatenate([np.arange(n), np.empty(n - 1, int)])
    out = {}
    for i, (a, b, h, s) in enumerate(Z):
        smallest[n + i] = min(smallest[int(a)], smallest[int(b)])
        out[(int(smallest[n + i]), int(s))] = h
    return out


CASES = {
    "11x3": lambda: normal(11, 3, seed=1),
    "129x8": lambda: blobs(129, 8, seed=2),
    "900x32": lambda: normal(900, 32, seed=3),
    "700x40": lambda: normal(700, 40, seed=4),
    "1500x2": lambda: blobs(1500, 2, centers=4, noise=0.1, seed=5),
    "far from the origin": lambda: (normal(600, 5, seed=6) + 3000).astype(f4),
    "ties": lambda: grid(24),
    "duplicates": lambda: np.repeat(normal(60, 4, seed=7), 9, axis=0),
    "more duplicates than a list": lambda: np.random.default_rng(7).permutation(
        np.repeat(normal(12, 4, seed=7), 40, axis=0)),
    "uneven sizes": lambda: np.vstack([normal(900, 3, seed=8) * f4(0.01),
                                       normal(60, 3, seed=9) * f4(20)]),
}


@pytest.mark.parametrize("screen", ["on", "off"])
@pytest.mark.parametrize("name", CASES)
def test_rounds_match_full_searches(name, screen):
    X = np.ascontiguousarray(CASES[name]())
    expected = clusters(ward_rounds(X), len(X))
    _lib.set_screen(screen)
    try:
        got = tree_clusters(_ward_rnn_with_options(X, min_progress=0.0))
    finally:
        _lib.set_screen("auto")
    assert got.keys() == expected.keys()
    keys = sorted(expected)
    np.testing.assert_allclose([got[k] for k in keys], [expected[k] for k in keys],
                               rtol=4 * 2.0 ** -23, atol=0)


@pytest.mark.parametrize("screen", ["on", "off"])
@pytest.mark.parametrize("name", CASES)
def test_kept_lists_match_full_searches(name, screen):
    """The same with lists kept down to the last clusters, as the default keeps them
    above a few thousand."""
    X = np.ascontiguousarray(CASES[name]())
    expected = clusters(ward_rounds(X), len(X))
    _lib.set_screen(screen)
    try:
        tree, rounds = _ward_rnn_with_lists(X, lists_above=1)
        full, none = _ward_rnn_with_lists(X, lists_above=len(X))
    finally:
        _lib.set_screen("auto")
    assert none == 0 and rounds >= (4 if len(X) > 100 else 1)
    np.testing.assert_array_equal(tree, full)
    got = tree_clusters(tree)
    assert got.keys() == expected.keys()
    keys = sorted(expected)
    np.testing.assert_allclose([got[k] for k in keys], [expected[k] for k in keys],
                               rtol=4 * 2.0 ** -23, atol=0)


HARD = {
    "heavy tails": lambda r: r.standard_t(1.5, (5000, 6)),
    "nested scales": lambda r: np.cumsum(r.standard_normal((12, 400, 9))
                                         * 0.1 ** np.arange(12)[:, None, None], 0).reshape(-1, 9),
    "nearly equal gaps": lambda r: np.arange(4000.0)[:, None] + r.uniform(-1e-4, 1e-4, (4000, 1)),
    "coarse far from the origin": lambda r: r.standard_normal((4000, 3)) + 4e4,
    "quantised": lambda r: r.integers(0, 5, (4500, 5)),
    "two chunks": lambda r: r.standard_normal((4000, 50)),
    "tiny values": lambda r: r.standard_normal((3000, 4)) * 1e-15,
    "huge values": lambda r: r.standard_normal((3000, 4)) * 1e16,
}


@pytest.mark.parametrize("screen", ["on", "off"])
@pytest.mark.parametrize("name", HARD)
def test_kept_lists_equal_full_searches(name, screen):
    """Larger sets, whose rounds have many clusters: bit for bit against the rounds
    that search every cluster (which the oracle above checks)."""
    X = np.ascontiguousarray(HARD[name](np.random.default_rng(5)), dtype=f4)
    _lib.set_screen(screen)
    try:
        tree, rounds = _ward_rnn_with_lists(X, lists_above=1)
        full, none = _ward_rnn_with_lists(X, lists_above=len(X))
    finally:
        _lib.set_screen("auto")
    assert none == 0 and rounds >= 4
    np.testing.assert_array_equal(tree, full)
