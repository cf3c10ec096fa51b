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
