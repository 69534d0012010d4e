"""Feature passes on host arrays of 64 MB of neighbours and more go slice by slice, each
with index staging of its own rows' size (csrc/capi.cu, csrc/features.cu): bit for bit the
device call's, for rows of one length and of several."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [30, (0, 61)])
def test_slices_equal_whole(cuda, pgeof, lengths):
    n = 600_001
    rng = np.random.default_rng(9)
    xyz = rng.random((50_000, 3), dtype=np.float32)
    counts = np.full(n, lengths) if isinstance(lengths, int) else rng.integers(*lengths, n)
    ptr = np.r_[0, np.cumsum(counts)].astype(np.uint32)
    nn = rng.integers(0, len(xyz), int(ptr[-1])).astype(np.uint32)
    assert nn.nbytes >= 64 << 20
    t_xyz, t_nn, t_ptr = (cuda.from_numpy(a).cuda() for a in (xyz, nn.view(np.int32), ptr.view(np.int32)))
    same = lambda host, dev: np.array_equal(host.view(np.uint32), dev.cpu().numpy().view(np.uint32))
    assert same(pgeof.compute_features(xyz, nn, ptr), pgeof.compute_features(t_xyz, t_nn, t_ptr))
    for scales in ([10, 30], [6, 10, 20, 30]):
        assert same(pgeof.compute_features_multiscale(xyz, nn, ptr, scales),
                    pgeof.compute_features_multiscale(t_xyz, t_nn, t_ptr, scales))
