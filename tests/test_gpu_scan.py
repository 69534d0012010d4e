"""The scan of cell counts (csrc/grid.cu) through radius_search_csr, whose row
pointers are such a scan over the queries: about a tile, and about the number of
tiles from which the tiles' sums are scanned by a kernel of their own."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 1023, 1024, 1025, 262_145, 4096 * 1024, 4096 * 1024 + 1])
def test_row_pointers(cuda, pgeof, m):
    g = cuda.Generator(device="cuda").manual_seed(5)
    x = cuda.rand((2000, 3), device="cuda", generator=g)
    q = cuda.rand((m, 3), device="cuda", generator=g)
    idx, _ = pgeof.radius_search(x, q, 0.04, 4)
    nn, ptr = pgeof.radius_search_csr(x, q, 0.04, 4)
    count = (idx.view(cuda.int32) >= 0).sum(1)
    assert int(ptr.view(cuda.int32)[0]) == 0
    assert cuda.equal(ptr.view(cuda.int32)[1:].long(), count.cumsum(0))
    assert cuda.equal(nn.view(cuda.int32), idx.view(cuda.int32)[idx.view(cuda.int32) >= 0])
