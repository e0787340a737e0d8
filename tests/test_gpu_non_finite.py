"""GPU: points without finite distances are refused under cosine.

Device arrays and the C entry points are not checked on the host. A row with an
infinite coordinate, or rows whose norms overflow, have NaN cosine distances; no
list pass may take one for an edge, whatever its route (k-NN lists, kept lists of
the rounds, radix select, min_samples 1 where the point itself is the only entry,
batches), below and above the feature counts of the tensor-core screen.
"""

import ctypes

import numpy as np
import pytest

import cuhc_b200 as C
from _data import normal
from cuhc_b200 import _batch, _lib  # noqa: F401 - _batch declares the batched entry
from cuhc_b200._hdbscan import hdbscan_tree

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

COSINE = C.METRIC_IDS["cosine"]


def infinite_row(d):
    X = normal(700, d, seed=d)
    X[17, d // 2] = np.inf
    return X


def overflowing_norms(d):
    return normal(700, d, seed=d) * np.float32(1e25)


@pytest.fixture(params=[infinite_row, overflowing_norms], ids=lambda f: f.__name__)
def points(request):
    return request.param


@pytest.mark.parametrize("d", [8, 48])
def test_single_linkage(points, d):
    with pytest.raises(RuntimeError, match="finite"):
        C.linkage(torch.from_numpy(points(d)).cuda(), "single", metric="cosine")


@pytest.mark.parametrize("d", [8, 48])
def test_single_linkage_host_entry(points, d):
    X, tree = points(d), np.empty((699, 4))
    assert _lib.lib.cuhc_linkage(_lib.float_ptr(X), 700, d, COSINE, 2.0, 0, 1,
                                 _lib.double_ptr(tree)) < 0


@pytest.mark.parametrize("d", [8, 48])
@pytest.mark.parametrize("k, method", [(1, "auto"), (5, "auto"), (1, "radix"), (300, "radix")])
def test_hdbscan(points, d, k, method):
    with pytest.raises(RuntimeError, match="finite"):
        hdbscan_tree(torch.from_numpy(points(d)).cuda(), k, metric="cosine", core_method=method)


@pytest.mark.parametrize("rank", [0, 1, 12])
def test_batch(points, rank):
    X = torch.from_numpy(np.vstack([normal(300, 8, seed=1), points(8)])).cuda()
    offsets, ranks = np.array([0, 300, 1000], np.int64), np.array([rank, rank], np.int32)
    tree, core = np.empty((998, 4)), np.empty(1000, np.float32)
    run = _lib.lib.cuhc_trees_batched_device
    run.argtypes = [ctypes.c_void_p, *_lib.lib.cuhc_trees_batched.argtypes[1:]]
    status = run(X.data_ptr(), _lib.int64_ptr(offsets), 2, 8, COSINE, 2.0,
                 ranks.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), _lib.double_ptr(tree),
                 _lib.float_ptr(core))
    assert status < 0

