"""GPU: calls of different sizes in several threads at once.

One kernel serves many sizes, each with its own amount of dynamic shared memory,
and the limit of that is shared by the process: no thread's call may fail because
another thread launches the same kernel with less, and results stay those of calls
made alone.
"""

import threading

import numpy as np
import pytest

import cuhc_b200 as C
from _data import normal
from cuhc_b200 import _lib
from cuhc_b200._hdbscan import hdbscan_tree

pytestmark = pytest.mark.gpu


def run_together(calls, repeats):
    """Every call, `repeats` times in a thread of its own, against its result alone."""
    expected = [call() for call in calls]
    failures = []

    def work(call, result):
        try:
            for _ in range(repeats):
                np.testing.assert_array_equal(call(), result)
        except Exception as error:  # noqa: BLE001 - reported in the main thread
            failures.append(error)

    threads = [threading.Thread(target=work, args=pair) for pair in zip(calls, expected)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not failures, failures


def test_distance_matrices_of_one_and_several_chunks():
    run_together([lambda X=normal(200, d, seed=d): C.pairwise_distances(X)
                  for d in (20, 32, 40, 64)], 400)


def test_dense_linkage_of_several_sizes():
    run_together([lambda X=normal(n, 3, seed=n): C.linkage(X, "average")
                  for n in (20, 130, 300, 520)], 100)


@pytest.mark.parametrize("screen", ["on", "off"])
def test_lists_of_several_lengths(screen):
    _lib.set_screen(screen)
    try:
        run_together([lambda X=normal(400, 7, seed=k), k=k: hdbscan_tree(X, k)[0]
                      for k in (1, 10, 40, 200)], 60)
    finally:
        _lib.set_screen("auto")
