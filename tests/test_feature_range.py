"""The feature ranges behind the float32 range check, around the 64-row blocks."""

import numpy as np
import pytest

from cuhc_b200._distances import _feature_range, check_distance_range


@pytest.mark.parametrize("n", [1, 63, 64, 65, 200, 4096])
@pytest.mark.parametrize("d", [1, 8, 70])
def test_feature_range(n, d):
    X = np.random.default_rng(n + d).standard_normal((n, d)).astype(np.float32)
    low, high = _feature_range(X)
    np.testing.assert_array_equal(low, X.min(axis=0))
    np.testing.assert_array_equal(high, X.max(axis=0))


@pytest.mark.parametrize("row", [0, 64, 99])
def test_one_far_row_is_seen(row):
    X, Y = np.zeros((100, 3), np.float32), np.zeros((5, 3), np.float32)
    X[row, 1] = -3e19
    for args in ({}, {"Y": Y}):
        with pytest.raises(ValueError, match="too large"):
            check_distance_range(X, "euclidean", **args)
    with pytest.raises(ValueError, match="too large"):
        check_distance_range(Y, "cosine", Y=X)
