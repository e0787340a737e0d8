"""GPU: the distance matrix at the edges of its kernel: output rows that do and
do not start on 16-byte boundaries (vector and scalar stores), tile remainders,
one, two and four feature chunks, an output that is itself unaligned. Bit for
bit against the CPU oracle."""

import ctypes

import numpy as np
import pytest

import cuhc_b200 as C
from _data import normal
from cuhc_b200 import _lib
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["euclidean", "manhattan", "cosine"])
@pytest.mark.parametrize("d", [1, 8, 33, 100])
@pytest.mark.parametrize("n, m", [(1, 4), (5, 3), (127, 128), (130, 129), (200, 260), (129, 258)])
def test_bits(n, m, d, metric):
    X, Y = normal(n, d, seed=n), normal(m, d, seed=m + 1000)
    np.testing.assert_array_equal(C.pairwise_distances(X, Y, metric=metric),
                                  O.pairwise(X, Y, metric=metric))


def test_unaligned_output():
    torch = pytest.importorskip("torch")
    X = torch.from_numpy(normal(140, 9, seed=3)).cuda()
    room = torch.full((140 * 140 + 1,), -1.0, device="cuda")
    _lib.check(_lib.lib.cuhc_pairwise_distances_device(
        X.data_ptr(), 140, None, 140, 9, 0, ctypes.c_float(2.0), room.data_ptr() + 4))
    np.testing.assert_array_equal(room[1:].cpu().numpy().reshape(140, 140),
                                  O.pairwise(X.cpu().numpy()))
    assert room[0].item() == -1.0
