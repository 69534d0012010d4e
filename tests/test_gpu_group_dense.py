"""Grouped search where a radius carried from a sparse place meets a dense one:
its staging is given up before the points are counted (csrc/group.cu). A batch of
such clouds against each cloud searched in slices, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 20, 100])
def test_dense_within_sparse(cuda, pgeof, k):
    rng = np.random.default_rng(41)
    sparse = rng.random((70_000, 3)) * [200.0, 200.0, 20.0]
    dense = rng.random((60_000, 3)) * [0.8, 0.8, 0.2] + [100.0, 100.0, 10.0]
    line = np.c_[rng.random((30_000, 1)) * 3.0, np.zeros((30_000, 2))] + [20.0, 150.0, 3.0]
    clouds = [np.concatenate([sparse, dense]), np.concatenate([sparse[:30_000], line]), dense]
    clouds = [cuda.from_numpy(c.astype(np.float32)).cuda() for c in clouds]
    idx, d2, _ = pgeof.batch_knn_features(clouds, k)
    at = 0
    for c in clouds:
        for a in range(0, c.shape[0], 50_000):
            i, d = pgeof.knn_search(c, c[a:a + 50_000].contiguous(), k)
            rows = slice(at + a, at + a + i.shape[0])
            assert cuda.equal(d2[rows].view(cuda.int32), d.view(cuda.int32))
            assert cuda.equal(idx[rows].view(cuda.int32), i.view(cuda.int32))
        at += c.shape[0]
