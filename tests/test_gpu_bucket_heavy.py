"""Sorts of inputs with one key that repeats about as often as a bucket has room for, and much more
often: seen in the sample (whole, or by 32 of its bits), found when its bucket overflows, or not too
frequent at all, for one and two partition steps; the largest key among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 4096


@pytest.mark.parametrize("bits", [30, 38, 60])
@pytest.mark.parametrize("n", [20_000, 300_000, 720_001, 3_000_001])
@pytest.mark.parametrize("copies", [1000, CAP, CAP + 1, 2 * CAP, 3 * CAP, None])
def test_one_heavy_key(cuda, n, bits, copies):
    rng = np.random.default_rng(n + bits)
    copies = n // 2 if copies is None else copies
    for top in (False, True):
        x = rng.integers(0, 1 << bits, size=n, dtype=np.uint64)
        x[rng.permutation(n)[:copies]] = np.uint64(2**64 - 1) if top else x[0]
        got, passes = cuda.sort(cuda.to_device(x))
        assert np.array_equal(cuda.to_numpy(got), np.sort(x))
        if copies == 1000 or copies > CAP:
            assert (passes > 3) == (copies > CAP)
        assert np.array_equal(cuda.to_numpy(cuda.unique(got)), np.unique(x))


@pytest.mark.parametrize("n", [50_000, 3_000_001])
def test_few_distinct_keys(cuda, n):
    x = np.random.default_rng(n).integers(0, 3, size=n, dtype=np.uint64) << np.uint64(40)
    got, _ = cuda.sort(cuda.to_device(x))
    assert np.array_equal(cuda.to_numpy(got), np.sort(x))
