"""Grouped searches large enough for their leftovers to be put in spatial order (csrc/group.cu,
csrc/search.cu): bit for bit the one-query search of the same queries in slices."""

import pytest

from point_geometric_features_gb300.synthetic import outdoor_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [799_999, 800_000, 1_600_003])
def test_large(cuda, pgeof, n):
    x = cuda.from_numpy(outdoor_scene(n, seed=101, box=(126.0, 126.0, 25.0), n_walls=60, n_cylinders=300)).cuda()
    for search in (lambda q: pgeof.knn_search(x, q, 12), lambda q: pgeof.radius_search(x, q, 0.3, 20)):
        idx, d2 = search(x)
        for a in range(0, n, 140_000):
            i, d = search(x[a : a + 140_000].contiguous())
            assert cuda.equal(d2[a : a + 140_000].view(cuda.int32), d.view(cuda.int32))
            assert cuda.equal(idx[a : a + 140_000].view(cuda.int32), i.view(cuda.int32))
