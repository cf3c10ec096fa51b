"""Sizes of the sort by buckets (csrc/bucketplan.h) on the host: every number of keys up to the stated
limit has a plan, whose buckets have room for what is expected of them, whose fine buckets one
partition step tells apart, and whose 32-bit offsets hold."""
import math
import os
import shutil
import subprocess

import pytest

from helpers import ROOT

TARGET, CAP, FAN, SAMPLES = 1800, 4096, 512, 8192


def test_every_size_up_to_the_limit_has_a_plan(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, "-std=c++17", "-O2", os.path.join(ROOT, "tests", "host", "bucket_plan_check.cu"), "-o", exe],
                   check=True, capture_output=True)

    def plans(ns):
        out = subprocess.run([exe] + [str(n) for n in ns], capture_output=True, text=True, check=True).stdout.split("\n")
        return int(out[0]), [tuple(map(int, line.split())) for line in out[1:] if line]

    limit, _ = plans([])
    ns = [2, CAP, CAP + 1, 400 * TARGET, 400 * TARGET + 1, limit - 1, limit]
    ns += [int(400 * TARGET * (limit / (400 * TARGET)) ** (i / 400)) for i in range(401)]  # and evenly over the logarithm
    for n, ok, coarse, cap, grid, words in plans(ns)[1]:
        assert ok, n
        assert grid * CAP < 1 << 32 and coarse * cap < 1 << 32, n
        if not coarse:
            assert n <= 400 * TARGET and grid * TARGET >= min(n, TARGET), n
            continue
        assert coarse <= FAN and cap <= FAN * TARGET, n
        assert cap >= n / coarse * (1 + 7 / math.sqrt(min(64, SAMPLES / coarse))) - 1, n
        assert grid >= n / TARGET + coarse - 1 and words >= 3 * FAN + 2 * grid, n
    assert [ok for _, ok, *_ in plans([limit + 1])[1]] == [0]
