"""What the fast forms hand on, made to happen: layer steps whose guesses were wrong (more spawns than
there was room for, more keys than the one CTA sorts that was expected to do), against the steps
that wait for every size (sort_variant 3), and sorts that go to the digit passes over 8192-key tiles
because one key repeats too often, around the edges of a tile."""
import numpy as np
import pytest

from cablegen_b200 import configs
from helpers import realistic_boards

pytestmark = pytest.mark.gpu

SMALL = 16384  # keys one CTA sorts


@pytest.fixture
def whole(cuda):
    """boards without fixed cells, nothing pruned: the most moves and spawns a board can have"""
    cuda.set_rules(configs.get("plain_2x4_nearwall").settings)
    return cuda


def boards(seed, n, p_empty):
    return np.unique(realistic_boards(np.random.default_rng(seed), n, formation_cells=(), p_empty=p_empty))


def moves(cuda, x):
    """(raw moves, the layer) of input boards"""
    raw = cuda.expand_moves(cuda.to_device(x))
    return raw.numel(), cuda.sort_unique(raw)


def same_as_with_waits(cuda, x, layers):
    end = 100 + 2 * (layers - 1)
    got, _ = cuda.generate(x, 100, end)
    cuda.set_option("sort_variant", 3)
    try:
        want, _ = cuda.generate(x, 100, end)
    finally:
        cuda.set_option("sort_variant", 4)
    assert sorted(got) == sorted(want) and len(got) == layers
    for s in want:
        assert len(want[s]) and np.array_equal(got[s], want[s]), s


def test_more_spawns_than_room(whole):
    x = boards(1, 5000, 0.75)
    _, layer = moves(whole, x)
    assert whole.count_spawns(layer) > 1.5 * len(x) * 16
    same_as_with_waits(whole, x, 2)


def test_spawns_beyond_the_one_cta_sort_expected(whole):
    for p in np.arange(0.20, 0.70, 0.01):
        x = boards(2, 800, p)
        _, layer = moves(whole, x)
        if whole.count_spawns(layer) > SMALL:
            break
    assert 1.25 * len(x) * 16 <= SMALL < whole.count_spawns(layer) <= 1.5 * len(x) * 16
    same_as_with_waits(whole, x, 2)


def test_moves_beyond_the_one_cta_sort_expected(whole):
    live = boards(3, 1000, 0.5)
    dead = np.uint64(0x1212212112122121)   # neighbours differ: no move
    x = np.concatenate([live, np.full(100_000, dead, np.uint64)])
    raw, layer = moves(whole, x)
    assert raw < 0.25 * len(x)   # the ratio that the next step expects
    two, _ = whole.expand_spawns(layer)
    inputs = whole.to_numpy(whole.sort_unique(two))
    assert 1.25 * len(inputs) * 0.25 <= SMALL < moves(whole, inputs)[0]
    same_as_with_waits(whole, x, 3)


@pytest.mark.parametrize("n", [2 * 8192 + 1, 3 * 8192 - 1, 3 * 8192, 3 * 8192 + 1, 25 * 8192, 1_000_003])
def test_repeats_go_to_digit_passes(cuda, n):
    x = np.random.default_rng(n).integers(0, 1 << 56, size=n, dtype=np.uint64) | np.uint64(0xFF << 56)
    x[::2] = x[0]
    got, passes = cuda.sort(cuda.to_device(x))
    assert passes == 7   # the varying bytes
    assert np.array_equal(cuda.to_numpy(got), np.sort(x))
