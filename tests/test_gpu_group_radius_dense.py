"""Grouped radius search (csrc/group.cu) where a sphere holds far more points than a group
can stage, in parts or at all, within a sparser cloud: bit for bit the one-query search of
the same queries in slices."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dense", [1_500, 20_000, 110_000])
def test_radius_in_dense_places(cuda, pgeof, dense):
    rng = np.random.default_rng(51)
    sparse = rng.random((180_000 - dense, 3)) * [60.0, 60.0, 3.0]
    spot = rng.normal(size=(dense, 3)) * 0.05 + [30.0, 30.0, 1.5]
    x = cuda.from_numpy(np.concatenate([sparse, spot])[rng.permutation(180_000)].astype(np.float32)).cuda()
    for r, k in ((0.6, 4), (0.6, 30), (0.02, 30), (0.6, 100)):
        idx, d2 = pgeof.radius_search(x, x, r, k)
        nn, ptr = pgeof.radius_search_csr(x, x, r, k)
        for a in range(0, x.shape[0], 60_000):
            i, d = pgeof.radius_search(x, x[a : a + 60_000].contiguous(), r, k)
            assert cuda.equal(d2[a : a + 60_000].view(cuda.int32), d.view(cuda.int32)), (r, k)
            assert cuda.equal(idx[a : a + 60_000].view(cuda.int32), i.view(cuda.int32)), (r, k)
        has = idx.view(cuda.int32) >= 0
        assert cuda.equal(nn.view(cuda.int32), idx.view(cuda.int32)[has])
        assert cuda.equal(ptr.view(cuda.int32)[1:].long(), has.sum(1).cumsum(0))
