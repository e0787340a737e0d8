"""GPU: calls go on without the arrays that only save time when there is no memory
for them (lists kept for the rounds, packed copies of rows), to the same results.
The limit stands in for memory that ran out: both take the same way."""

import numpy as np
import pytest

import cuhc_b200 as C
from _data import blobs, normal
from cuhc_b200 import _lib
from cuhc_b200._hdbscan import hdbscan_tree

pytestmark = pytest.mark.gpu

N, D = 3000, 32
# No array at all; the lists (9 entries of 4 bytes a point) and no copy of the rows.
LIMITS = {"nothing": 0, "lists only": 24 * 128 * 9 * 4}

CALLS = {
    "single": lambda: (C.linkage(normal(N, D, seed=1), "single"),),
    "single, several chunks": lambda: (C.linkage(normal(N, 40, seed=1), "single", "cosine"),),
    "hdbscan": lambda: hdbscan_tree(normal(N, D, seed=2), 9),
    "ward": lambda: (C.linkage(normal(N, D, seed=3), "ward"),),
    "batch": lambda: [a for pair in C.batched_trees(
        [normal(n, D, seed=n) for n in (700, 1300, 5)], [0, 9, 2]) for a in pair],
}


@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("name", CALLS)
def test_same_results_without(name, limit):
    CALLS[name]()  # tuners have run
    before = _lib.launch_count()
    expected = CALLS[name]()
    usual = _lib.launch_count() - before
    _lib.set_optional_memory(LIMITS[limit])
    try:
        before = _lib.launch_count()
        got = CALLS[name]()
        without = _lib.launch_count() - before
    finally:
        _lib.set_optional_memory(None)
    assert without != usual  # it did take another way
    for a, b in zip(got, expected):
        np.testing.assert_array_equal(a, b)


def test_a_large_limit_changes_nothing():
    X = blobs(2500, 8, seed=4)
    before = _lib.launch_count()
    expected = C.linkage(X, "single")
    usual = _lib.launch_count() - before
    _lib.set_optional_memory(1 << 30)
    try:
        before = _lib.launch_count()
        np.testing.assert_array_equal(C.linkage(X, "single"), expected)
        assert _lib.launch_count() - before == usual
    finally:
        _lib.set_optional_memory(None)
