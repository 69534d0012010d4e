"""Feature passes of one process over rows of different lengths: how much shared memory
stays L1 (cap_smem_carveout, csrc/capi.cu) is each launch's own choice, whatever was
launched before. A pass over 50 neighbours a row, then over 56, 60, 64, 72: fewer
neighbours take no longer than more. (Where a launch ran under the wrong choice it took
1.6 times as long as the next longer rows.)"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scales", [None, [10, 30], [10, 20, 30]])
def test_shorter_rows_are_no_slower(cuda, pgeof, scales):
    n, widths = 500_000, (50, 56, 60, 64, 72)
    g = cuda.Generator(device="cuda").manual_seed(3)
    xyz = cuda.rand((n, 3), device="cuda", generator=g)
    nn = cuda.randint(0, n, (n * max(widths),), device="cuda", generator=g, dtype=cuda.int32)
    ms = []
    for k in widths:
        ptr = cuda.arange(0, k * (n + 1), k, dtype=cuda.int32, device="cuda")
        times = []
        for _ in range(7):
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            if scales:
                pgeof.compute_features_multiscale(xyz, nn[: n * k], ptr, scales + [k], check=False)
            else:
                pgeof.compute_features(xyz, nn[: n * k], ptr, check=False)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms.append(sorted(times)[3])
    for shorter, longer in zip(ms, ms[1:]):
        assert shorter <= 1.25 * longer, ms
