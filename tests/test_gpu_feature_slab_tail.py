"""A last warp of one, two or three long rows of one even length behind many short ones,
whose indices still fit the staging of csrc/features.cu, against the oracle. The lengths
are ones for which a reciprocal multiply in 22 bits is not the division by the row length.
Same tolerance as test_gpu_features.py."""

import numpy as np
import pytest

from conftest import align_normals, feature_close
from oracle import oracle

pytestmark = pytest.mark.gpu


def csr(short, n_short, tail, n_tail, whole_mean):
    """n_short rows of `short` neighbours and n_tail of `tail`, each of whose last neighbour
    is far from the rest; with `whole_mean` some of the first rows get one more, until the
    mean row length is a whole number."""
    counts = np.r_[np.full(n_short, short), np.full(n_tail, tail)]
    if whole_mean:
        counts[: -int(counts.sum()) % len(counts)] += 1
    rng = np.random.default_rng(5)
    xyz = (rng.random((4000, 3)) * [1.0, 0.6, 0.3]).astype(np.float32)
    xyz[7] = [4.0, -3.0, 5.0]
    ptr = np.r_[0, np.cumsum(counts)].astype(np.uint32)
    nn = rng.integers(8, len(xyz), int(ptr[-1])).astype(np.uint32)
    nn[ptr[-1 - n_tail :][1:] - 1] = 7
    return xyz, nn, ptr


@pytest.mark.parametrize("whole_mean", [False, True])
@pytest.mark.parametrize("short,n_short,tail,n_tail", [(70, 64, 3000, 1), (5, 32, 4000, 1), (2, 32, 2094, 1), (70, 64, 1506, 2),
                                                       (5, 32, 1506, 2), (70, 64, 1230, 3), (2, 32, 1300, 3)])
def test_long_last_rows(cuda, pgeof, short, n_short, tail, n_tail, whole_mean):
    xyz, nn, ptr = csr(short, n_short, tail, n_tail, whole_mean)
    rows = np.diff(ptr) >= 5
    ref = oracle.compute_features(xyz, nn, ptr, 1)
    got = pgeof.compute_features(xyz, nn, ptr, 1)
    assert feature_close(align_normals(got[rows], ref[rows]), ref[rows]).all()
    scales = [5, tail // 2, tail]
    ref = oracle.compute_features_multiscale(xyz, nn, ptr, scales)
    got = pgeof.compute_features_multiscale(xyz, nn, ptr, scales)
    assert feature_close(align_normals(got[rows], ref[rows]), ref[rows]).all()


@pytest.mark.parametrize("whole_mean", [False, True])
@pytest.mark.parametrize("tail,n_tail", [(2094, 1), (2162, 1), (1506, 2), (1230, 3)])
def test_long_last_rows_several_scales(cuda, pgeof, tail, n_tail, whole_mean):
    """As above with rows enough for the staging to serve several scales."""
    xyz, nn, ptr = csr(120 if n_tail > 1 else 70, 20_000, tail, n_tail, whole_mean)
    tail_ptr = ptr[-1 - n_tail :]
    for scales in ([5, tail], [5, 60, tail], [5, 20, 60, tail]):
        got = pgeof.compute_features_multiscale(xyz, nn, ptr, scales)[-n_tail:]
        ref = oracle.compute_features_multiscale(xyz, nn[tail_ptr[0] :], (tail_ptr - tail_ptr[0]).astype(np.uint32), scales)
        assert feature_close(align_normals(got, ref), ref).all(), scales
