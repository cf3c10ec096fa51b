"""An FP32 sweep's FP64 window reaches the caller whole: its tables are narrowed and given back while
copies of them may still be on their way, behind callbacks that take their time.  Every window table is
compared bit for bit with the FP64 sweep's; the FP32 tables below stay within 1e-6 of it."""
import ctypes as C
import time

import numpy as np
import pytest

from cablegen_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,end", [("plain_2x4_nearwall", 120), ("dpdf", 380)])
def test_fp64_window_tables_are_whole(cuda, name, end):
    w = configs.get(name)
    f = w.formations[0]
    cuda.set_rules(w.settings)
    top = cuda.get_option("fp64_top_layers")
    assert top == 4
    low = end - 2 * (top + 3)  # the window and three FP32 layers

    def sweep(precision):
        got = {}

        def on_table(s, keys, vals, n, prec):
            v = np.ctypeslib.as_array(C.cast(vals, C.POINTER(C.c_double if prec == 64 else C.c_float)), shape=(n,))
            time.sleep(0.002)
            got[s] = (prec, v.copy())

        cuda.tablebase(f.initial, f.start, end, low, f.winstates, precision=precision, table_fn=on_table)
        return got

    want = sweep(64)
    for _ in range(5):
        got = sweep(32)
        assert sorted(got) == sorted(want)
        for s, (prec, v) in got.items():
            if s > end - 2 * top:
                assert prec == 64 and np.array_equal(v, want[s][1]), s
            else:
                assert prec == 32 and np.abs(v - want[s][1]).max() <= 1e-6, s
