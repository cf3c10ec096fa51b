"""The look-back wait of the bucket sort made to run out on purpose: its first bucket does not publish its
count, so that with the poll limit lowered every later one gives up and reports it.  Sorts that keep
repeats (one and two partition steps) and those that drop them (a layer step); the same context
sorts correctly afterwards."""
import numpy as np
import pytest

from cablegen_b200 import _lib, configs
from helpers import realistic_boards

pytestmark = pytest.mark.gpu


@pytest.fixture
def held(cuda):
    assert cuda.get_option("sort_variant") == 4
    try:
        cuda.set_option("lookback_spin_limit", 4096)
        cuda.set_option("lookback_hold_first_tile", 1)
        yield
    finally:
        cuda.set_option("lookback_hold_first_tile", 0)
        cuda.set_option("lookback_spin_limit", 0)


@pytest.mark.parametrize("n", [20_000, 300_000, 1_500_000])
def test_sort_wait_runs_out(cuda, held, n):
    x = np.random.default_rng(n).integers(0, 1 << 40, size=n, dtype=np.uint64)
    t = cuda.to_device(x)
    with pytest.raises(_lib.CablegenError, match="look-back wait timed out"):
        cuda.sort(t)
    cuda.set_option("lookback_hold_first_tile", 0)
    assert np.array_equal(cuda.to_numpy(cuda.sort(t)[0]), np.sort(x))


def test_layer_step_wait_runs_out(cuda, held):
    cuda.set_rules(configs.get("ll_pruned").settings)
    x = np.unique(realistic_boards(np.random.default_rng(5), 60_000))
    with pytest.raises(_lib.CablegenError, match="look-back wait timed out"):
        cuda.generate(x, 100, 100)
    cuda.set_option("lookback_hold_first_tile", 0)
    got, _ = cuda.generate(x, 100, 100)
    moves = cuda.expand_moves(cuda.to_device(x))
    assert moves.numel() > 16384 and np.array_equal(got[100], np.unique(cuda.to_numpy(moves)))
