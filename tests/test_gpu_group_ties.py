"""Grouped search of grids, where nearly every distance ties and the k-th with some that
are kept and some that are not (csrc/group.cu: order_ties): lattices, a flat one, a voxelised
scene, each with and without duplicates; bit for bit the one-query search of the same queries
in slices, a sample against the oracle."""

import numpy as np
import pytest

from oracle import oracle
from point_geometric_features_gb300.synthetic import outdoor_scene

pytestmark = pytest.mark.gpu


def grid(kind):
    if kind == "lattice":
        p = np.stack(np.meshgrid(*[np.arange(56)] * 3), -1).reshape(-1, 3) * 0.5
    elif kind == "flat":
        p = np.stack(np.meshgrid(np.arange(500), np.arange(340), [3]), -1).reshape(-1, 3) * 0.25
    elif kind == "flat twice":
        p = np.repeat(np.stack(np.meshgrid(np.arange(330), np.arange(260), [3]), -1).reshape(-1, 3), 2, 0) * 0.25
    else:
        p = np.round(outdoor_scene(400_000, seed=81, box=(60.0, 60.0, 12.0), n_walls=10, n_cylinders=50) / 0.05)
        if kind == "voxels":
            p = np.unique(p, axis=0)
        p = p[:180_000] * 0.05 if kind == "voxels, repeated" else p * 0.05
    return np.random.default_rng(82).permutation(p.astype(np.float32))


@pytest.mark.parametrize("kind", ["lattice", "flat", "flat twice", "voxels", "voxels, repeated"])
def test_grid(cuda, pgeof, kind):
    x = grid(kind)
    assert len(x) >= 150_000
    t = cuda.from_numpy(x).cuda()
    rows = np.random.default_rng(1).choice(len(x), 60, replace=False)
    step = float(np.sort(np.unique(x[:, 0]))[1] - np.sort(np.unique(x[:, 0]))[0])
    knn = [(pgeof.knn_search, oracle.knn_search, (k,)) for k in (1, 2, 5, 7, 9, 19, 27, 33, 50, 64)]
    radius = [(pgeof.radius_search, oracle.radius_search, (m * step, k)) for m, k in ((1.01, 4), (2.3, 10), (2.3, 64), (4.1, 30))]
    for search, ref, args in knn + radius:
        idx, d2 = search(t, t, *args)
        for a in range(0, len(x), 70_000):
            i, d = search(t, t[a : a + 70_000].contiguous(), *args)
            assert cuda.equal(d2[a : a + 70_000].view(cuda.int32), d.view(cuda.int32)), args
            assert cuda.equal(idx[a : a + 70_000].view(cuda.int32), i.view(cuda.int32)), args
        ri, rd = ref(x, x[rows], *args)
        np.testing.assert_array_equal(idx.view(cuda.int32)[rows].cpu().numpy(), ri.view(np.int32))
        np.testing.assert_array_equal(d2[rows].cpu().numpy(), rd)
