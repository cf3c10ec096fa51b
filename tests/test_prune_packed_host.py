"""prune_packed (board.cuh: every count of the prune rule in one u64 per byte) against prune_board on
the host: the parameter sets of the workloads, both ends of the smallest_large range it takes, and
limits that every board or no board passes; other parameters leave it off."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import ROOT, realistic_boards

ON = [(58, 5, 6), (64, 6, 6), (200, 5, 5), (0, 0, 6), (-64, 3, 7), (58, 5, 13), (58, 5, 14), (30, 3, 8), (10**6, 40, 5),
      (1000, 31, 12), (511 - 64, 16, 5), (512 - 64, 15, 6)]
OFF = [(58, 5, 4), (58, 5, -1), (58, 5, 15), (-65, 5, 6), (58, -1, 6)]


def test_packed_prune(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, "-std=c++17", "-O2", os.path.join(ROOT, "tests", "host", "prune_packed_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    rng = np.random.default_rng(3)
    np.concatenate([
        realistic_boards(rng, 20000, max_exp=13, p_empty=0.2),
        realistic_boards(rng, 20000, formation_cells=(), max_exp=8, p_empty=0.1),
        rng.integers(0, 1 << 63, 20000, dtype=np.uint64) * np.uint64(2),
        np.array([int("".join(rng.choice(list("5556667789"), 16)), 16) for _ in range(5000)], dtype=np.uint64),
        np.array([int(c * 16, 16) for c in "0123456789abcdef"], dtype=np.uint64)]).tofile(tmp_path / "b.u64")
    sets = ON + OFF
    r = subprocess.run([exe, str(tmp_path / "b.u64")] + [",".join(map(str, p)) for p in sets], capture_output=True, text=True,
                       check=True)
    for p, line in zip(sets, r.stdout.strip().split("\n")):
        on, _, _, bad = map(int, line.split())
        assert on == (p in ON) and bad == 0, (p, line)
