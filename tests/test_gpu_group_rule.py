"""Which searches go by groups (csrc/group.cuh, csrc/grid.cu): surfaces and volumes, k and
numbers of queries about the rule's lines, sparse and dense radii, and an index whose calls
differ from the ones its cells were sized for. Whatever way a call takes, the rows are those
of the same queries in slices, bit for bit; a sample against the oracle."""

import numpy as np
import pytest

from oracle import oracle
from point_geometric_features_gb300.synthetic import outdoor_scene, uniform_cube

pytestmark = pytest.mark.gpu


def clouds(n):
    side = (n / 100) ** 0.5
    yield outdoor_scene(n, seed=71, box=(side, side, side / 5), n_walls=8, n_cylinders=40)
    yield uniform_cube(n, seed=72)
    line = np.zeros((n, 3), np.float32)
    line[:, 0] = np.random.default_rng(73).random(n)
    yield line


def same_rows(cuda, search, got, q):
    for a in range(0, q.shape[0], 70_000):
        part = search(q[a : a + 70_000].contiguous())
        for g, p in zip(got, part):
            assert cuda.equal(g[a : a + 70_000].view(cuda.int32), p.view(cuda.int32))


@pytest.mark.parametrize("m", [149_999, 150_000, 199_999, 200_000, 225_000, 300_000])
@pytest.mark.parametrize("k", [1, 64, 65, 100, 101])
def test_knn(cuda, pgeof, m, k):
    for x in clouds(300_000):
        t = cuda.from_numpy(x).cuda()
        q = t[:m].contiguous() + 0.001
        got = pgeof.knn_search(t, q, k)
        same_rows(cuda, lambda s: pgeof.knn_search(t, s, k), got, q)
        rows = cuda.arange(0, m, m // 40, device="cuda")
        ri, rd = oracle.knn_search(x, q[rows].cpu().numpy(), k)
        np.testing.assert_array_equal(got[1][rows].cpu().numpy(), rd)
        np.testing.assert_array_equal(got[0].view(cuda.int32)[rows].cpu().numpy().astype(np.uint32), ri)


def test_knn_many_neighbours(cuda, pgeof):
    for x in clouds(500_000):
        t = cuda.from_numpy(x).cuda()
        same_rows(cuda, lambda s: pgeof.knn_search(t, s, 128), pgeof.knn_search(t, t, 128), t)


@pytest.mark.parametrize("k", [8, 40, 64, 80, 128])
@pytest.mark.parametrize("found", [2, 8, 20, 60])
def test_radius(cuda, pgeof, found, k):
    n = 210_000
    for x, r in zip(clouds(n), ((found / 157) ** 0.5, (found / n / 4.19) ** (1 / 3), found / n / 2)):
        t = cuda.from_numpy(x).cuda()
        same_rows(cuda, lambda s: pgeof.radius_search(t, s, r, k), pgeof.radius_search(t, t, r, k), t)


def test_index(cuda, pgeof):
    for x in clouds(220_000):
        t = cuda.from_numpy(x).cuda()
        for hints in ({}, {"k_hint": 50}, {"k_hint": 100}, {"k_hint": 32, "radius_hint": 0.05}):
            ix = pgeof.GridIndex(t, **hints)
            for k in (5, 90):
                for q in (None, t[:1000].contiguous(), t[:160_000].contiguous() + 0.002):
                    a, b = ix.knn_search(q, k), pgeof.knn_search(t, t if q is None else q, k)
                    assert all(cuda.equal(u.view(cuda.int32), v.view(cuda.int32)) for u, v in zip(a, b))
                a, b = ix.radius_search(None, 0.05, k), pgeof.radius_search(t, t, 0.05, k)
                assert all(cuda.equal(u.view(cuda.int32), v.view(cuda.int32)) for u, v in zip(a, b))
