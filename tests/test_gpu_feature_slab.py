"""Feature passes whose rows' indices are staged in shared memory (features.cu):
row lengths about a warp's width and the staging's limit, ragged rows, partial
last warps, against the oracle. Same tolerance as test_gpu_features.py."""

import numpy as np
import pytest

from conftest import align_normals, feature_close
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rows", [1, 31, 32, 33, 129, 1000])
@pytest.mark.parametrize("k", [8, 31, 32, 33, 50, 64, 127, 128, 129, "ragged"])
def test_row_lengths(cuda, pgeof, n_rows, k):
    rng = np.random.default_rng(11)
    xyz = rng.random((5000, 3), dtype=np.float32)
    counts = rng.integers(0, 90, n_rows) if k == "ragged" else np.full(n_rows, k)
    ptr = np.r_[0, np.cumsum(counts)].astype(np.uint32)
    nn = rng.integers(0, xyz.shape[0], int(ptr[-1])).astype(np.uint32)
    top = 89 if k == "ragged" else k
    for scales in ([top], [5, top], [3, 8, top], [3, 5, 7, top], [1, 2, 3, 4, 5, 6, 7, top]):
        ref = oracle.compute_features_multiscale(xyz, nn, ptr, scales)
        got = pgeof.compute_features_multiscale(xyz, nn, ptr, scales)
        # (fewer than 5 points: repeated zero eigenvalues, whose eigenvectors are free)
        keep = [q for q, size in enumerate(scales) if size >= 5]
        got, ref = got[:, keep], ref[:, keep]
        assert feature_close(align_normals(got, ref), ref).all()
        assert ((got == 0).all(axis=-1) == (ref == 0).all(axis=-1)).all()
    ref = oracle.compute_features(xyz, nn, ptr, 1)
    got = pgeof.compute_features(xyz, nn, ptr, 1)
    rows = counts >= 5
    assert feature_close(align_normals(got[rows], ref[rows]), ref[rows]).all()
