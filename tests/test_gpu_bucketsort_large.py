"""The sort by buckets on inputs up to its limit: three passes (two partition steps and the buckets'
sort) where the plan needs as many coarse buckets as fine ones in each, where it needs more of them,
and at the limit; digit passes one key above it.  Keys of 12 and of 8 cells that vary, as a layer's do."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LIMIT = 160 << 20


@pytest.mark.parametrize("n,bits", [(99_092_495, 48), (99_092_496, 32), (120_000_001, 48), (LIMIT, 48), (LIMIT + 1, 32)])
def test_large_sort(cuda, n, bits):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randint(0, 1 << bits, (n,), generator=g, device="cuda", dtype=torch.int64)
    got, passes = cuda.sort(x)
    assert (passes == 3) == (n <= LIMIT), passes
    assert torch.equal(got, torch.sort(x).values)
