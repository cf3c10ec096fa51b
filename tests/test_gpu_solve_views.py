"""The board-pair solve with one lane per view, which small layers take, against the same boards solved
as part of a large layer (all views in one lane): bit for bit, layer sizes around the limits (two
boards for each of the chip's 4736 warps, one a warp up to 4736), tables with NaN values included."""
import numpy as np
import pytest
import torch

from cablegen_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layers(cuda):
    w = configs.get("ll_pruned", end_gen=170)
    f = w.formations[0]
    cuda.set_rules(w.settings)
    got, _ = cuda.generate(f.initial, f.start, f.end_gen)
    return w, [got[s] for s in (166, 168, 170)]


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 4736, 4737, 9472, 9473])
def test_small_layer_matches_part_of_large(cuda, layers, n, precision):
    w, (now, s2, s4) = layers
    assert len(now) > 2 * 9473
    cuda.set_rules(w.settings)
    rng = np.random.default_rng(n)
    dt = np.float64 if precision == 64 else np.float32
    tables = []
    for k in (s2, s4):
        v = rng.random(len(k)).astype(dt)
        v[::101] = np.nan
        tables.append((cuda.to_device(k), torch.from_numpy(v).cuda()))
    pick = np.sort(rng.choice(len(now), n, replace=False))

    def solve(keys):
        return cuda.solve_layer(cuda.to_device(keys), *tables, w.formations[0].winstates,
                                precision=precision).cpu().numpy()

    want = solve(now)
    assert np.isnan(want).any()
    assert np.array_equal(solve(now[pick]), want[pick], equal_nan=True)
