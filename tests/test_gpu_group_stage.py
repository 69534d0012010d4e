"""Grouped search of volumes, whose groups need the most candidates (csrc/group.cu): every k
about which the room for them changes, over the points themselves and over fewer queries,
and radii that find from few to many times what is kept; bit for bit the one-query search
of the same queries in slices."""

import pytest

pytestmark = pytest.mark.gpu


def check(cuda, search, x, q):
    idx, d2 = search(x, q)
    for a in range(0, q.shape[0], 60_000):
        i, d = search(x, q[a : a + 60_000].contiguous())
        assert cuda.equal(d2[a : a + 60_000].view(cuda.int32), d.view(cuda.int32))
        assert cuda.equal(idx[a : a + 60_000].view(cuda.int32), i.view(cuda.int32))


@pytest.fixture(scope="module")
def volume(cuda):
    g = cuda.Generator(device="cuda").manual_seed(61)
    return cuda.rand((230_000, 3), device="cuda", generator=g), cuda.rand((175_000, 3), device="cuda", generator=g)


@pytest.mark.parametrize("k", [1, 3, 8, 15, 16, 17, 24, 33, 49, 51, 63, 64, 65, 81, 100, 101, 127, 128])
def test_volume(cuda, pgeof, volume, k):
    x, q = volume
    check(cuda, lambda a, b: pgeof.knn_search(a, b, k), x, x)
    check(cuda, lambda a, b: pgeof.knn_search(a, b, k), x, q)


@pytest.mark.parametrize("k", [1, 10, 33, 64, 100, 128])
@pytest.mark.parametrize("found", [4, 30, 180, 700])
def test_radius(cuda, pgeof, volume, found, k):
    x, _ = volume
    r = (found / x.shape[0] / 4.19) ** (1 / 3)
    check(cuda, lambda a, b: pgeof.radius_search(a, b, r, k), x, x)
