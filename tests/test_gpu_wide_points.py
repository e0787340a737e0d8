"""GPU: points of so many features that a block's shared memory holds them but no
k-NN lists beside them. Calls that need no lists run without; the trees are those
of the oracle, or of the dense algorithm."""

import numpy as np
import pytest

import cuhc_b200 as C
from _data import assert_same_dendrogram, blobs
from cuhc_b200._linkage import _ward_rnn_with_lists
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# Lists of 9 entries leave room for about 19,000 features, none for about 20,100.
WIDE = 19_800


@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_single_linkage(metric):
    X = blobs(300, WIDE, seed=1)
    np.testing.assert_array_equal(C.linkage(X, "single", metric=metric),
                                  O.single_linkage(X, metric=metric))


def test_batch():
    instances = [blobs(n, WIDE, seed=n) for n in (40, 150)]
    for (Z, core), X in zip(C.batched_trees(instances, [0, 0]), instances):
        np.testing.assert_array_equal(Z, O.single_linkage(X))
        assert not core.any()


def test_ward():
    X = blobs(2100, WIDE, centers=40, seed=2)
    assert_same_dendrogram(C.linkage(X, "ward"), C.linkage(X, "ward", algorithm="dense"))
    tree, listed = _ward_rnn_with_lists(X, lists_above=500)
    assert listed == 0  # asked for, but there is no room
    np.testing.assert_array_equal(tree, C.linkage(X, "ward"))
