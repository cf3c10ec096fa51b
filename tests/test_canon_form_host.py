"""The three closed forms of a canonical plan (board.cuh: canon_form) against the full canonical
form on the host: every formation of the plan test in all eight orientations and all four views;
LL, 2x4 and DPDF take the form their fixed cells allow."""
import os
import shutil
import subprocess

import pytest

from helpers import ROOT
from test_canon_plan_host import FORMATIONS, cellmask

LIST, ONE, DIAGONAL, MIRROR = range(4)


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    out = str(tmp_path_factory.mktemp("host") / "canon_form_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", os.path.join(ROOT, "tests", "host", "canon_form_check.cu"), "-o", out],
                   check=True, capture_output=True)
    return out


@pytest.mark.parametrize("name,form", [("LL", DIAGONAL), ("2x4", MIRROR), ("DPDF", ONE), ("centre", LIST)]
                         + [(n, None) for n in FORMATIONS if n not in ("LL", "2x4", "DPDF", "centre")])
def test_forms_give_the_canonical_board(checker, name, form):
    r = subprocess.run([checker, f"{cellmask(FORMATIONS[name]):04x}"], capture_output=True, text=True, check=True)
    for line in r.stdout.strip().split("\n"):
        _, got, checked, bad = (int(x, 16 if i == 0 else 10) for i, x in enumerate(line.split()))
        assert bad == 0 and checked == (0 if got == LIST else 20000), line
        assert form is None or got == form, line
