"""The grouped search (searches of 150k queries and more, csrc/group.cu) against the
one-query-per-warp search of the same queries in slices, bit for bit, and against the
oracle on a sample: clouds with surfaces, volumes, exact ties, duplicates and far
queries; k at the edges of its range; radii that find fewer and more than max_knn."""

import numpy as np
import pytest

from oracle import oracle
from point_geometric_features_gb300.synthetic import outdoor_scene, uniform_cube

pytestmark = pytest.mark.gpu

SLICE = 50_000  # below the grouped search's smallest number of queries


def cloud(kind):
    if kind == "scene":
        return outdoor_scene(200_003, seed=21, box=(45.0, 45.0, 9.0), n_walls=8, n_cylinders=40)
    if kind == "volume":
        return uniform_cube(150_001, seed=22)
    if kind == "ties":  # a voxel grid, some voxels taken twice
        rng = np.random.default_rng(23)
        return (np.floor(rng.random((160_000, 3)) * [90, 90, 12]) * 0.25).astype(np.float32)
    rng = np.random.default_rng(24)  # "clusters": densities orders of magnitude apart, and an offset
    centre = rng.random((40, 3)) * 50.0 + 1000.0
    spread = 10.0 ** rng.uniform(-2.5, 0.5, 40)
    at = rng.integers(0, 40, 170_001)
    return (centre[at] + rng.normal(size=(170_001, 3)) * spread[at, None]).astype(np.float32)


def in_slices(fn, q):
    parts = [fn(q[a:a + SLICE].contiguous()) for a in range(0, q.shape[0], SLICE)]
    import torch

    return [torch.cat([p[j].view(torch.int32) for p in parts]) for j in range(2)]


@pytest.mark.parametrize("kind,ks", [("scene", (1, 2, 16, 33, 64, 65, 128)), ("volume", (8, 50)), ("ties", (5, 30)),
                                     ("clusters", (10, 40))])
def test_grouped_knn_equals_sliced(cuda, pgeof, kind, ks):
    x = cloud(kind)
    t = cuda.from_numpy(x).cuda()
    rows = np.random.default_rng(1).choice(len(x), 200, replace=False)
    for k in ks:
        idx, d2 = pgeof.knn_search(t, t, k)
        i2, e2 = in_slices(lambda q: pgeof.knn_search(t, q, k), t)
        assert cuda.equal(d2.view(cuda.int32), e2), (kind, k)
        assert cuda.equal(idx.view(cuda.int32), i2), (kind, k)
        ri, rd = oracle.knn_search(x, x[rows], k)
        np.testing.assert_array_equal(d2[rows].cpu().numpy(), rd)
        np.testing.assert_array_equal(idx.view(cuda.int32)[rows].cpu().numpy().astype(np.uint32), ri)


@pytest.mark.parametrize("kind,r,ks", [("scene", 0.3, (1, 16, 64)), ("scene", 0.8, (30, 128)), ("volume", 0.05, (64,)),
                                       ("ties", 0.6, (12,)), ("clusters", 0.05, (20,)), ("volume", 1e-12, (4,))])
def test_grouped_radius_equals_sliced(cuda, pgeof, kind, r, ks):
    x = cloud(kind)
    t = cuda.from_numpy(x).cuda()
    for k in ks:
        idx, d2 = pgeof.radius_search(t, t, r, k)
        i2, e2 = in_slices(lambda q: pgeof.radius_search(t, q, r, k), t)
        assert cuda.equal(idx.view(cuda.int32), i2), (kind, r, k)
        assert cuda.equal(d2.view(cuda.int32), e2), (kind, r, k)
        nn, ptr = pgeof.radius_search_csr(t, t, r, k)
        has = idx >= 0
        assert cuda.equal(nn.view(cuda.int32), idx[has])
        assert cuda.equal(ptr.view(cuda.int32)[1:].long(), has.sum(1).cumsum(0))


def test_grouped_external_queries(cuda, pgeof):
    """More queries than points, some of them far outside the cloud."""
    x = cloud("scene")[:120_000]
    q = outdoor_scene(180_000, seed=31, box=(45.0, 45.0, 9.0), n_walls=8, n_cylinders=40)
    q[::1000] += np.float32(500.0)
    q[1::1000, 2] -= np.float32(300.0)
    t, tq = cuda.from_numpy(x).cuda(), cuda.from_numpy(q).cuda()
    idx, d2 = pgeof.knn_search(t, tq, 12)
    i2, e2 = in_slices(lambda s: pgeof.knn_search(t, s, 12), tq)
    assert cuda.equal(d2.view(cuda.int32), e2) and cuda.equal(idx.view(cuda.int32), i2)
    idx, d2 = pgeof.radius_search(t, tq, 0.7, 20)
    i2, e2 = in_slices(lambda s: pgeof.radius_search(t, s, 0.7, 20), tq)
    assert cuda.equal(d2.view(cuda.int32), e2) and cuda.equal(idx.view(cuda.int32), i2)
