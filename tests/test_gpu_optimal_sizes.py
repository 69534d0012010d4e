"""compute_features_optimal where sizes tie or are many (csrc/features.cu): more near-tied
sizes than a row keeps, more sizes than the scan ranks, rows that are lines, planes,
duplicates or a voxel grid. The size found has the smallest float64 eigentropy up to the
rounding of the float formula (its terms are below 1 and hold ~10 roundings of 6e-8 each:
2e-6), and the features are compute_features' own for that size."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows_of(kind, n, k, rng):
    """n rows of k points each, as a cloud of n * k points."""
    if kind == "voxel":  # many exact ties, few different directions
        p = np.round(rng.random((n, k, 3)) * [3.0, 3.0, 0.6])
    elif kind == "plane":
        p = rng.random((n, k, 3)) * [1.0, 1.0, 0.0]
    elif kind == "line":
        p = rng.random((n, k, 1)) * np.array([1.0, 2.0, -0.5])
    elif kind == "duplicates":  # one point, then another one
        p = np.repeat(rng.random((n, 1, 3)), k, 1)
        p[:, 2 * k // 3 :] += 0.25
    elif kind == "steady":  # a square walked round: every fourth size is the same shape
        p = np.tile(np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]], float), (n, (k + 3) // 4, 1))[:, :k]
        p = p + rng.random((n, 1, 3))
    else:
        p = rng.random((n, k, 3)) * [1.0, 0.5, 0.2]
    return p.astype(np.float32)


def eigentropy64(p, sizes):
    """float64 eigentropies (include/pca.hpp:140-150) of the first k points, k in sizes, of every row."""
    out = []
    for k in sizes:
        q = p[:, :k].astype(np.float64)
        q = q - q.mean(1, keepdims=True)
        w = np.maximum(np.linalg.eigvalsh(np.einsum("nki,nkj->nij", q, q) / k), 0.0)
        e = w / (w.sum(1, keepdims=True) + 1e-3)
        out.append(-(e * np.log(e + 1e-3)).sum(1))
    return np.stack(out, 1)


@pytest.mark.parametrize("n", [3, 700, 6000])
@pytest.mark.parametrize("kind", ["random", "voxel", "plane", "line", "duplicates", "steady"])
@pytest.mark.parametrize("k,step", [(20, 1), (73, 1), (74, 1), (110, 1), (110, 7), (75, 64)])
def test_optimal_size(cuda, pgeof, kind, n, k, step):
    p = rows_of(kind, n, k, np.random.default_rng(k + step))
    xyz = p.reshape(-1, 3)
    nn = np.arange(n * k, dtype=np.uint32)
    ptr = np.arange(0, n * k + 1, k, dtype=np.uint32)
    got = pgeof.compute_features_optimal(xyz, nn, ptr, 1, step, 10)
    sizes = [s for s in range(10, k + 1) if s == 10 or s % step == 0 or s == k]
    found = got[:, 11].astype(int)
    assert np.isin(found, sizes).all()
    ent = eigentropy64(p, sizes)
    at = np.searchsorted(sizes, found)
    assert (ent[np.arange(n), at] <= ent.min(1) + 2e-6).all()
    cut = np.concatenate([nn[r * k : r * k + found[r]] for r in range(n)])
    assert np.array_equal(got[:, :11], pgeof.compute_features(xyz, cut, np.r_[0, np.cumsum(found)].astype(np.uint32), 1))
