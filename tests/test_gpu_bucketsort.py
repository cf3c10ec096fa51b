"""The sort by sampled buckets (csrc/bucketsort.cu) against numpy at the sizes where it changes
form -- one bucket (up to 4096 and up to 16384 keys), one partition step (up to 400 x 1800 keys), two steps -- for
keys whose buckets differ in the low word alone, in at most 32 bits of both words, and in more; keys
with repeats; and inputs it hands on to the digit passes (a bucket that cannot hold its repeats)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ONE, SMALL, TWO = 4096, 16384, 400 * 1800


def keys(kind, n):
    rng = np.random.default_rng(n + len(kind))
    if kind == "low":       # one high word
        return rng.integers(0, 1 << 32, size=n, dtype=np.uint64) | np.uint64(0xABCD << 40)
    if kind == "nibbles":   # twelve cells of three bits: 36 bits spread over both words
        x = np.zeros(n, np.uint64)
        for c in range(12):
            x |= rng.integers(0, 8, size=n, dtype=np.uint64) << np.uint64(4 * c + 8)
        return x | np.uint64(0xFF)
    if kind == "wide":      # all 64 bits
        return rng.integers(0, 1 << 63, size=n, dtype=np.uint64) * np.uint64(2) + rng.integers(0, 2, size=n).astype(np.uint64)
    if kind == "repeats":   # about three copies of each key, the largest value among them
        return ~(rng.integers(0, max(n // 3, 1), size=n, dtype=np.uint64) << np.uint64(20))
    if kind == "sorted":
        return np.sort(rng.integers(0, 1 << 40, size=n, dtype=np.uint64))
    x = rng.integers(0, 1 << 50, size=n, dtype=np.uint64)
    x[: n // 2] = 5         # "heavy": half of the input is one key
    return x


@pytest.mark.parametrize("kind", ["low", "nibbles", "wide", "repeats", "sorted", "heavy"])
@pytest.mark.parametrize("n", [2, 15, 17, 511, 513, 2049, ONE, ONE + 1, 9001, SMALL, SMALL + 1, TWO, TWO + 1, 3_000_017])
def test_bucket_sort(cuda, kind, n):
    x = keys(kind, n)
    got, _ = cuda.sort(cuda.to_device(x))
    want = np.sort(x)
    assert np.array_equal(cuda.to_numpy(got), want)
    assert np.array_equal(cuda.to_numpy(cuda.sort_unique(cuda.to_device(x))), np.unique(x))
