"""cgb_lookup_batch by search of the sorted layer and through the hash index against numpy: layers
around the sizes where a search changes its number of steps, board counts on both sides of each
form's range (a warp per board, a thread per board, the index), the smallest and largest keys."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1024, 1025, 1057, 70001])
def test_lookup_forms(cuda, n, precision):
    rng = np.random.default_rng(n)
    keys = np.unique(rng.integers(1, 1 << 63, size=n, dtype=np.uint64) * np.uint64(2) - np.uint64(1))
    if n > 2:
        keys[-1] = ~np.uint64(0)
    vals = rng.random(len(keys)).astype(np.float64 if precision == 64 else np.float32)
    k, v = cuda.to_device(keys), torch.from_numpy(vals).cuda()
    for m in sorted({1, 5, len(keys), len(keys) + 1, 4096, 4097, 60000}):
        q = keys[rng.integers(0, len(keys), m)]
        q = np.where(rng.random(m) < 0.3, q - np.uint64(1), q)   # not members: keys are odd
        q[0] = keys[0] - np.uint64(1)                             # below every key
        if m > 3:
            q[1], q[2], q[3] = keys[0], keys[-1], np.uint64(2)
        at = np.minimum(np.searchsorted(keys, q), len(keys) - 1)
        want = np.where(keys[at] == q, vals[at].astype(np.float64), 0.0)
        got = cuda.lookup_batch(k, v, cuda.to_device(q)).cpu().numpy()
        assert np.array_equal(got, want), (n, m)
