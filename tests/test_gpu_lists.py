"""GPU: the Borůvka rounds that search only some of the rows.

Single linkage and HDBSCAN keep every point's nearest few; later rounds settle
rows from those lists, leave out rows whose bound exceeds their component's
best, let large components sit rounds out, and pack the remaining rows into
row tiles of their own where boxes exclude little, splitting few row tiles
over the columns. Every tree must equal the CPU oracle's bit for bit: at list
lengths around the point count, with ties at the last list entry, with
components above and below the sizes that sit out, packed through the
per-instance and the device-wide selection, screened and plain, one feature
chunk and several.
"""

import numpy as np
import pytest

import cuhc_b200 as C
from _data import blobs, grid, normal
from cuhc_b200 import _lib
from cuhc_b200._hdbscan import hdbscan_tree
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["on", "off"], ids=["screened", "plain"])
def screen(request):
    _lib.set_screen(request.param)
    yield
    _lib.set_screen("auto")


CASES = {
    "2x2": lambda: normal(2, 2, seed=1),
    "8x3": lambda: normal(8, 3, seed=2),
    "9x3": lambda: normal(9, 3, seed=3),
    "10x3": lambda: normal(10, 3, seed=4),
    "129x5": lambda: normal(129, 5, seed=5),
    "grid": lambda: grid(45),
    "duplicates": lambda: np.repeat(blobs(250, 4, seed=6), 12, axis=0),
    "far apart": lambda: blobs(6000, 2, centers=3, noise=0.2, seed=7, std=(0.1, 0.2)),
    "chain": lambda: np.cumsum(np.linspace(1, 2, 3000))[:, None].astype(np.float32),
    "packed": lambda: normal(5000, 32, seed=8),
    "packed, device-wide select": lambda: normal(16_500, 20, seed=9),
    "two chunks": lambda: normal(3000, 40, seed=10),
    # Enough points for lists in plain passes.
    "large grid": lambda: grid(65),
    "many duplicates": lambda: np.repeat(blobs(250, 4, seed=13), 18, axis=0),
    "long chain": lambda: np.cumsum(np.linspace(1, 2, 4200))[:, None].astype(np.float32),
    "two chunks, packed": lambda: normal(4100, 40, seed=14),
    # More row tiles than start at once: large components sit rounds out in place.
    "sitting out in place": lambda: blobs(38_100, 2, centers=3, noise=0.2, seed=12),
}


@pytest.mark.parametrize("name", CASES)
def test_single_linkage(screen, name):
    X = CASES[name]()
    np.testing.assert_array_equal(C.linkage(X, "single"), O.single_linkage(X))


@pytest.mark.parametrize("n, d, k", [(3000, 32, 10), (3000, 40, 5), (6000, 2, 40)])
def test_hdbscan(screen, n, d, k):
    X = normal(n, d, seed=k) if d > 2 else blobs(n, d, centers=3, noise=0.2, seed=k)
    Z, core = hdbscan_tree(X, k)
    Z_ref, core_ref = O.hdbscan_tree(X, k)
    np.testing.assert_array_equal(core, core_ref)
    np.testing.assert_array_equal(Z, Z_ref)


def test_batch_of_sitting_out_components(screen):
    """Instances far apart in size, in one solve, in place and packed."""
    for d in (2, 32):
        instances = [blobs(n, d, centers=2, seed=n) for n in (5, 4000, 130, 2500)]
        ranks = [0, 0, 7, 12]
        for (Z, core), X, k in zip(C.batched_trees(instances, ranks), instances, ranks):
            Z_ref, core_ref = O.hdbscan_tree(X, k) if k else (O.single_linkage(X), 0)
            np.testing.assert_array_equal(Z, Z_ref)
            np.testing.assert_array_equal(core, core_ref)


def test_nan_rows_stay_disconnected():
    """A point without finite distances: refused as before, lists or not."""
    torch = pytest.importorskip("torch")
    X = torch.from_numpy(normal(600, 8, seed=11)).cuda()
    X[17, 3] = float("nan")
    with pytest.raises(RuntimeError, match="finite"):
        C.linkage(X, "single")


@pytest.mark.parametrize("n, copies", [(300, 300), (900, 10), (900, 9), (1600, 200)])
@pytest.mark.parametrize("d, k", [(3, 9), (40, 1), (40, 12)])
def test_rows_done_early(screen, n, copies, d, k):
    """Lists of nothing but equal points, with a tie outside the list or not."""
    X = np.repeat(normal(n // copies, d, seed=d), copies, axis=0)
    X = np.random.default_rng(n).permutation(X)
    np.testing.assert_array_equal(C.linkage(X, "single"), O.single_linkage(X))
    Z, core = hdbscan_tree(X, k)
    Z_ref, core_ref = O.hdbscan_tree(X, k)
    np.testing.assert_array_equal(core, core_ref)
    np.testing.assert_array_equal(Z, Z_ref)
