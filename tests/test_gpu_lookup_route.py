"""Which way cgb_lookup_batch takes -- by search of the sorted layer or through an index, which the
statistics count -- on both sides of its lines, and the values either way."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

M = 1 << 20


@pytest.mark.parametrize("n,bits,most", [
    (2 * M, 32, 2 * M), (2 * M + 8, 32, 2 * M + 8 - 3 * (2 * M + 8) // 8), (4 * M, 32, 4 * M - 3 * M // 2), (4 * M + 4, 32, 3 * M + 3),
    (8 * M, 32, 6 * M), (8 * M + 1, 32, 8 * M + 1), (8 * M, 64, 8 * M), (8 * M + 5, 64, 8 * M + 5 - (8 * M + 5) // 5),
    (16 * M + 4, 64, 4 * M + 1), (16 * M + 4, 32, 4 * M + 1)])
def test_route_and_values(cuda, n, bits, most):
    g = torch.Generator(device="cuda").manual_seed(n + bits)
    keys = torch.unique(torch.randint(0, 1 << 48, (n + n // 64,), generator=g, device="cuda", dtype=torch.int64))[:n]
    assert keys.numel() == n
    vals = torch.rand(n, generator=g, device="cuda", dtype=torch.float64).to(torch.float64 if bits == 64 else torch.float32)
    at = torch.randint(0, n, (most + 1,), generator=g, device="cuda")
    boards = keys[at]
    boards[::7] += 1   # mostly not in the layer
    where = torch.searchsorted(keys, boards).clamp(max=n - 1)
    want = torch.where(keys[where] == boards, vals[where].double(), 0.0)
    for m, builds in ((most, 0), (most + 1, 1)):
        before = cuda.kernel_stats()["index_builds"]
        got = cuda.lookup_batch(keys, vals, boards[:m])
        assert cuda.kernel_stats()["index_builds"] - before == builds, m
        assert torch.equal(got, want[:m])
