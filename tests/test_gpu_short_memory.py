"""Calls under a cap on device memory that has room for what they need, though not for what would only
make them faster.  Each runs in a process of its own, where nothing is held yet."""
import subprocess
import sys
import textwrap

import pytest

from helpers import ROOT

pytestmark = pytest.mark.gpu

HEAD = """
    import ctypes as C, sys
    import numpy as np
    sys.path.insert(0, {root!r})
    sys.path.insert(0, {root!r} + "/tests")
    from cablegen_b200 import _lib, configs, device
    from helpers import realistic_boards
    import torch
    device.init(0)
    w = configs.get("ll_pruned")
    device.set_rules(w.settings)
"""


def run(body):
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(HEAD.format(root=ROOT)) + textwrap.dedent(body)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]


def test_layer_step_without_room_for_its_guess():
    """400K nearly full boards spawn about one each, but the first step's room is a guess of 16, 192 MB."""
    run("""
        x = np.unique(realistic_boards(np.random.default_rng(1), 400_000, p_empty=0.03))
        device.set_option("device_mem_cap_mb", 160)
        got, _ = device.generate(x, 100, 102)
        device.set_option("device_mem_cap_mb", 0)
        want, _ = device.generate(x, 100, 102)
        assert sorted(got) == sorted(want) == [100, 102]
        assert all(len(want[s]) > 100_000 and np.array_equal(got[s], want[s]) for s in want)
    """)


SOLVE = """
        x = np.unique(realistic_boards(np.random.default_rng(2), 1_500_000))[:1_000_000]
        many, few = device.to_device(x), device.to_device(x[:10])
        val = torch.rand(len(x), dtype=torch.float64, device="cuda")
        full, tiny = (many, val), (few, val[:10])
        f = w.formations[0]

        def solve(t2, t4):
            return device.solve_layer(many[::100].contiguous(), t2, t4, f.winstates).cpu().numpy()

        want = solve(tiny, full), solve(full, tiny)
"""


def test_kept_indexes_make_room():
    """Two one-layer solves, each with one large table (64 MB of slots and 28 MB of build scratch), one
    above and one below: what is kept from the first is in the way of the second."""
    run(SOLVE + """
        device.set_option("device_mem_cap_mb", 130)
        for _ in range(2):
            assert np.array_equal(solve(full, tiny), want[1])
            assert np.array_equal(solve(tiny, full), want[0])
            got = device.lookup_batch(few, val[:10], many[:40])   # more boards than keys: an index
            assert torch.equal(got[:10], val[:10]) and not got[10:].any()
    """)


@pytest.mark.parametrize("cap", [150, 210])
def test_sort_space_makes_room(cap):
    """A sort of 4M keys keeps its buckets (168 MB; under the lower cap it gets half of them and gives
    up), which are in the way of a one-layer solve that needs 92 MB."""
    run(SOLVE + """
        device.set_option("device_mem_cap_mb", 0)
        k = torch.randint(0, 1 << 48, (4_000_000,), device="cuda", dtype=torch.int64)
    """ + f"    device.set_option('device_mem_cap_mb', {cap})\n" + """
        for _ in range(2):
            assert torch.equal(device.sort(k)[0], torch.sort(k).values)
            assert np.array_equal(solve(full, tiny), want[1])
    """)


def test_cap_counts_what_was_kept_before_it():
    """Blocks that a sweep freed are kept for the next; a cap set afterwards gives them back, so that the
    engine holds what it says it holds, and a sweep under the cap stays below it."""
    run("""
        drv = C.CDLL("libcuda.so.1")
        pool = C.c_void_p()
        assert drv.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0

        def used():
            v = C.c_uint64()
            assert drv.cuMemPoolGetAttribute(pool, 7, C.byref(v)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
            return v.value

        f, peak = w.formations[0], []
        def sweep():
            device.tablebase(f.initial, f.start, 120, f.start, f.winstates,
                             table_fn=lambda *a: peak.append(used()))

        sweep()
        torch.cuda.synchronize()
        before = used()
        device.set_option("device_mem_cap_mb", 1)
        after = used()
        try:
            sweep()
            raise SystemExit("a sweep within 1 MB")
        except _lib.CablegenError as e:
            held = float(str(e).split("(")[1].split(" GB held")[0]) * 1e9
        small = 32 << 20  # the sort's own words are not counted
        assert after <= held + small, (before, after, held)
        cap = 4 << 30
        device.set_option("device_mem_cap_mb", cap >> 20)
        peak.clear()
        sweep()
        assert max(peak) <= cap + small, (max(peak), cap)
    """)
