"""Hash indexes filled by the solve itself against indexes built from keys and values, by region
and by atomic inserts: the tables below them are equal bit for bit (every index is exact), over
layers up to above the 2^16 keys that regions start at, 16- and 8-byte slots, sparse and
crowded slots."""
import numpy as np
import pytest

from cablegen_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,compact", [(64, 0), (32, 0), (32, 1)])
@pytest.mark.parametrize("load", [0, 90])
def test_filled_index_matches_built(cuda, precision, compact, load):
    w = configs.get("ll_pruned", end_gen=220)
    f = w.formations[0]
    cuda.set_rules(w.settings)
    names = ("solve_variant", "region_build", "hash_compact", "hash_load_pct")
    old = {k: cuda.get_option(k) for k in names}
    got = {}
    try:
        cuda.set_option("hash_compact", compact)
        cuda.set_option("hash_load_pct", load)
        for variant, region in ((1, 1), (0, 1), (0, 0)):  # filled, by region, by atomic inserts
            cuda.set_option("solve_variant", variant)
            cuda.set_option("region_build", region)
            _, got[variant, region], _ = cuda.tablebase(f.initial, f.start, f.end_gen, f.start, f.winstates,
                                                        precision=precision, keep_tables=True)
    finally:
        for k, v in old.items():
            cuda.set_option(k, v)
    sizes = [len(k) for k, _ in got[1, 1].values()]
    assert max(sizes) >= 1 << 16
    for other in ((0, 1), (0, 0)):
        for s, (_, vals) in got[1, 1].items():
            assert np.array_equal(got[other][s][1], vals), (other, s)
