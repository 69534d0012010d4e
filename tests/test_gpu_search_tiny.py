"""Searches at distances whose squares are near the smallest floats, with more candidates
than a warp's buffer holds, against the oracle: the bound that the candidates' histogram
gives (csrc/search.cu) has no scale there."""

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,r", [(1e-19, 4e-19), (1e-18, 1.5e-18), (1e-17, 1.5e-17)])
def test_radius(cuda, pgeof, side, r):
    rng = np.random.default_rng(7)
    x = (rng.random((2000, 3)) * side).astype(np.float32)
    idx, d2 = pgeof.radius_search(x, x, r, 10)
    ri, rd = oracle.radius_search(x, x, r, 10)
    np.testing.assert_array_equal(idx, ri)
    np.testing.assert_array_equal(d2, rd)


@pytest.mark.parametrize("extent", [1e-7, 1e-6, 1e-5])
def test_knn_cluster(cuda, pgeof, extent):
    """A cluster of 2,000 points 1e-20 wide within a cloud of `extent`."""
    rng = np.random.default_rng(8)
    x = np.concatenate([rng.random((3000, 3)) * extent, rng.random((2000, 3)) * 1e-20]).astype(np.float32)
    for k in (8, 40):
        idx, d2 = pgeof.knn_search(x, x, k)
        ri, rd = oracle.knn_search(x, x, k)
        np.testing.assert_array_equal(d2, rd)
        np.testing.assert_array_equal(idx, ri)
