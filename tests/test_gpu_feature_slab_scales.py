"""Several scales over rows enough for the index staging of csrc/features.cu (one block per
SM and more), with even, odd and unequal row lengths and a partial last warp: a sample of
the rows and all of the last warp against the oracle (tolerance of test_gpu_features.py),
and every row bit for bit against the same rows in slices too short for the staging."""

import numpy as np
import pytest

from conftest import align_normals, feature_close
from oracle import oracle

pytestmark = pytest.mark.gpu

SLICE = 9_000


def take_rows(nn, ptr, rows):
    counts = (ptr[1:] - ptr[:-1])[rows]
    part = np.concatenate([nn[ptr[r] : ptr[r + 1]] for r in rows]) if len(rows) else nn[:0]
    return part.astype(np.uint32), np.r_[0, np.cumsum(counts)].astype(np.uint32)


@pytest.mark.parametrize("n_rows", [20_011, 40_001])
@pytest.mark.parametrize("lengths", [16, 31, 32, 64, 65, 80, (0, 48), (0, 20)])
def test_scales(cuda, pgeof, n_rows, lengths):
    rng = np.random.default_rng(17)
    xyz = (rng.random((6000, 3)) * [1.0, 0.7, 0.4]).astype(np.float32)
    counts = np.full(n_rows, lengths) if isinstance(lengths, int) else rng.integers(*lengths, n_rows)
    top = int(counts.max())
    ptr = np.r_[0, np.cumsum(counts)].astype(np.uint32)
    nn = rng.integers(0, len(xyz), int(ptr[-1])).astype(np.uint32)
    sample = np.unique(np.r_[rng.choice(n_rows, 300, replace=False), n_rows - n_rows % 32 : n_rows])
    s_nn, s_ptr = take_rows(nn, ptr, sample)
    dev = lambda a: cuda.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()
    t_xyz, t_nn, t_ptr = dev(xyz), dev(nn), dev(ptr)
    for scales in ([8, top], [6, 9, top], [5, 6, 9, top], [5, 6, 7, 8, 9, top], [5, 6, 7, 8, 9, 10, 11, top]):
        got = pgeof.compute_features_multiscale(t_xyz, t_nn, t_ptr, scales)
        for a in range(0, n_rows, SLICE):
            b = min(a + SLICE, n_rows)
            part = pgeof.compute_features_multiscale(t_xyz, t_nn[int(ptr[a]) : int(ptr[b])].contiguous(),
                                                     t_ptr[a : b + 1] - int(ptr[a]), scales)
            assert cuda.equal(got[a:b].view(cuda.int32), part.view(cuda.int32)), (scales, a)
        ref = oracle.compute_features_multiscale(xyz, s_nn, s_ptr, scales)
        mine = got[cuda.from_numpy(sample).cuda()].cpu().numpy()
        assert feature_close(align_normals(mine, ref), ref).all(), scales
