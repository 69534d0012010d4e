"""Exact duplicates in numbers about a warp's candidate buffer (256 and 512 keys) and beyond,
alone and within a scene, against the oracle: the one-query search must not tighten for
ever (csrc/search.cu)."""

import numpy as np
import pytest

from oracle import oracle
from point_geometric_features_gb300.synthetic import outdoor_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [255, 257, 513, 1500, 5000])
def test_duplicates(cuda, pgeof, copies):
    rng = np.random.default_rng(11)
    places = np.repeat(rng.random((3, 3)) * [10.0, 10.0, 2.0], copies, 0)
    x = np.concatenate([places, outdoor_scene(3000, seed=12, box=(10.0, 10.0, 2.0), n_walls=4, n_cylinders=4)])
    x = x[rng.permutation(len(x))].astype(np.float32)
    rows = np.unique(np.r_[rng.choice(len(x), 150, replace=False), 0])
    for k in (1, 20, 100):
        idx, d2 = pgeof.knn_search(x, x, k)
        ri, rd = oracle.knn_search(x, x[rows], k)
        np.testing.assert_array_equal(d2[rows], rd)
        np.testing.assert_array_equal(idx[rows], ri)
    for r, k in ((0.01, 20), (0.8, 64)):
        idx, d2 = pgeof.radius_search(x, x, r, k)
        ri, rd = oracle.radius_search(x, x[rows], r, k)
        np.testing.assert_array_equal(d2[rows], rd)
        np.testing.assert_array_equal(idx[rows], ri)
