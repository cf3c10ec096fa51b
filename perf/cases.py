"""The work a user of the engine has it do, as cases that can be timed and compared.

Five kinds, over the workloads of cablegen_b200/configs.py:

* ``table``  -- a whole tablebase: generation from the initial boards, then the solve, every
  table delivered to the caller's host arrays (what the CLI's generate + solve is for).
* ``batch``  -- the same for many formations in one run.
* ``step``   -- one layer step through the device primitives: moves, sort, unique, the 2- and
  4-spawns, their sorts, and the merge into the next input set (a caller's own layer loop).
* ``solve``  -- one layer solved against the two tables above it.
* ``lookup`` -- positions looked up in a solved layer: a few (play, explore) or many (an
  evaluator, a training-data extractor).

Boards are real ones: whole sweeps from seeded initial boards, and contiguous slices of a
workload's layers for the kinds that take a layer.  ``exact`` computes values in float64 with
plain torch (its own row moves, canonical forms and searches).
"""
import ctypes
import math
import random

import numpy as np
import torch

from cablegen_b200 import _lib, configs, device

# --------------------------------------------------------------------------- cases
# Boards of a workload's tables from its start up to a tile sum (whole initial set).
CUMULATIVE = {
    "plain_2x4_nearwall": [(20, 600), (60, 31000), (100, 104000), (160, 205000), (220, 303000), (300, 392000)],
    "dpdf": [(312, 150000), (330, 2.2e6), (350, 8.0e6), (380, 2.13e7), (400, 3.2e7)],
    "ll_pruned": [(40, 1.2e5), (60, 1.4e6), (80, 7.5e6), (100, 1.9e7), (120, 4.3e7), (140, 7.1e7)],
    "ll_large": [(24, 1.3e5), (28, 1.3e6), (32, 6.5e6), (34, 1.2e7)],
}
# Sizes of one layer step per input board: layer, next input set and 4-spawn set.
STEP_OUT = {"plain_2x4_nearwall": 4.1, "dpdf": 3.3, "ll_pruned": 2.9, "ll_large": 12.0}


def listed():
    return [
        # the smallest tablebase anyone builds: 149 layers of a few thousand boards, all latency
        {"name": "table 2x4 fp64", "kind": "table", "workload": "plain_2x4_nearwall", "end": 300, "precision": 64},
        # ordinary: layers of about a million boards, FP32 tables
        {"name": "table dpdf fp32", "kind": "table", "workload": "dpdf", "end": 380, "precision": 32},
        # the flagship formation over its first 53 layers, FP64 as the reference solves it
        {"name": "table ll fp64", "kind": "table", "workload": "ll_pruned", "end": 120, "precision": 64},
        # free formation: 0xf cells move, all eight images can be canonical, many empty cells
        {"name": "table ll free fp64", "kind": "table", "workload": "ll_large", "end": 34, "precision": 64},
        # a dozen formations at once
        {"name": "batch 12 fp32", "kind": "batch", "formations": 12, "end": 200, "precision": 32},
        # one layer step: tiny, ordinary (odd size), large
        {"name": "step 2x4 1201", "kind": "step", "workload": "plain_2x4_nearwall", "sum": 64, "boards": 1201},
        {"name": "step dpdf 300007", "kind": "step", "workload": "dpdf", "sum": 380, "boards": 300007},
        {"name": "step ll 4000000", "kind": "step", "workload": "ll_pruned", "sum": 196, "boards": 4000000},
        # one layer solved: the flagship's size in FP64, an odd smaller one in FP32
        {"name": "solve ll 5000000 fp64", "kind": "solve", "workload": "ll_pruned", "sum": 196, "boards": 5000000,
         "precision": 64},
        {"name": "solve dpdf 250001 fp32", "kind": "solve", "workload": "dpdf", "sum": 380, "boards": 250001,
         "precision": 32},
        # an evaluator's million positions, and the hundred that play or explore asks for
        {"name": "lookup ll 1000003 fp64", "kind": "lookup", "workload": "ll_pruned", "sum": 196, "boards": 1000003,
         "precision": 64},
        {"name": "lookup dpdf 100 fp32", "kind": "lookup", "workload": "dpdf", "sum": 380, "boards": 100,
         "precision": 32},
    ]


# Tile sums at which a workload's layers hold more boards than the largest slice drawn from them.
SLICES = {"plain_2x4_nearwall": (40, 240, 200, 1500), "dpdf": (336, 400, 1000, 300000),
          "ll_pruned": (130, 196, 10000, 2000000), "ll_large": (28, 32, 5000, 600000)}
ENDS = {"plain_2x4_nearwall": (40, 300), "dpdf": (312, 380), "ll_pruned": (40, 120), "ll_large": (24, 34)}


def _even(rng, lo, hi):
    return 2 * rng.randint(lo // 2, hi // 2)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["table", "batch", "step", "solve", "lookup"])
    precision = rng.choice([64, 32])
    if kind == "batch":
        return {"kind": kind, "formations": _log(rng, 2, 16), "end": _even(rng, 100, 200), "precision": precision}
    workload = rng.choice(sorted(SLICES))
    if kind == "table":
        return {"kind": kind, "workload": workload, "end": _even(rng, *ENDS[workload]), "precision": precision}
    lo, hi, few, many = SLICES[workload]
    case = {"kind": kind, "workload": workload, "sum": _even(rng, lo, hi), "boards": _log(rng, few, many)}
    if kind == "lookup":
        case["boards"] = _log(rng, 1, 1000000)
    if kind != "step":
        case["precision"] = precision
    return case


def work(case):
    """Inputs read once and outputs written once."""
    value = case.get("precision", 64) // 8
    if case["kind"] == "table":
        pts = CUMULATIVE[case["workload"]]
        xs, ys = [p[0] for p in pts], [math.log(p[1]) for p in pts]
        boards = math.exp(float(np.interp(case["end"], xs, ys)))
        return {"bytes": boards * (8 + value), "flops": 0}
    if case["kind"] == "batch":
        return {"bytes": case["formations"] * max(case["end"] - 60, 20) * 27000.0 * (8 + value), "flops": 0}
    n = case["boards"]
    if case["kind"] == "step":
        return {"bytes": 8 * n * (1.5 + STEP_OUT[case["workload"]]), "flops": 0}
    if case["kind"] == "solve":  # the layer and its values; each table above it once
        return {"bytes": 3 * n * (8 + value), "flops": 0}
    return {"bytes": n * (8 + 8 + 8 + value), "flops": 0}


# --------------------------------------------------------------------------- inputs
def _workload(name):
    return configs.get(name)


def _subset(boards, rng, share):
    """A seeded part of a list of boards, in its order."""
    keep = sorted(rng.sample(range(len(boards)), max(1, round(len(boards) * share))))
    return [boards[i] for i in keep]


def _layers(case, sums):
    """The named layers of a workload on the GPU (generated from its whole initial set)."""
    w = _workload(case["workload"])
    f = w.formations[0]
    got = {}

    def keep(s, ptr, n):
        if s in sums:
            host = np.empty(n, np.int64)
            if n:
                ctypes.memmove(host.ctypes.data, ptr, 8 * n)
            got[s] = torch.from_numpy(host).cuda()

    # nothing is solved (the solve ends above the last layer); only the layers are kept
    device.tablebase(f.initial, f.start, max(sums), max(sums) + 2, [], layer_fn=keep)
    return w, [got[s] for s in sums]


def _slice(t, n, rng):
    at = rng.randrange(0, t.numel() - n + 1)
    return t[at:at + n].clone()


def _values(n, precision, gen):
    """Win probabilities: a share of the boards lost, the others spread over (0, 1)."""
    v = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    v = torch.where(torch.rand(n, generator=gen, device="cuda") < 0.1, torch.zeros_like(v), v)
    return v.to(torch.float32 if precision == 32 else torch.float64)


_SIGN = -(1 << 63)  # boards order as unsigned: the sign bit is turned over to compare them


def _unique(*parts):
    return torch.unique(torch.cat(parts) ^ _SIGN) ^ _SIGN


def prepare(case, seed):
    device.init(0)
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed & 0x7FFFFFFF)
    kind = case["kind"]
    if kind == "table":
        w = _workload(case["workload"])
        device.set_rules(w.settings)
        f = w.formations[0]
        # room for the tables of the whole initial set, which hold those of any part of it
        _, st = device.generate(f.initial, f.start, case["end"], keep=False)
        room = int(st["boards_generated"])
        dt = torch.float32 if case["precision"] == 32 else torch.float64
        # values come as FP64 for the highest layers of an FP32 sweep: kept apart
        initial = _subset(f.initial, rng, 0.3 if len(f.initial) <= 16 else 0.75)
        return {"case": case, "initial": initial, "start": f.start, "win": f.winstates,
                "keys": torch.empty(room, dtype=torch.int64).fill_(0), "vals": torch.empty(room, dtype=dt).fill_(0),
                "vals64": torch.empty(room if dt == torch.float32 else 1, dtype=torch.float64).fill_(0),
                "sizes": torch.zeros((case["end"] - f.start) // 2 + 1, dtype=torch.int64)}
    if kind == "batch":
        w = configs.batch64(n_formations=case["formations"])
        device.set_rules(w.settings)
        forms = []
        for f in w.formations:
            f.end_gen = min(f.end_gen, case["end"])
            forms.append(f)
        _, _, st = device.batch(forms, precision=case["precision"])
        room = int(st["boards_generated"])
        for f in forms:
            f.initial = _subset(f.initial, rng, 0.75)
        dt = torch.float32 if case["precision"] == 32 else torch.float64
        return {"case": case, "forms": forms, "keys": torch.empty(room, dtype=torch.int64).fill_(0),
                "vals": torch.empty(room, dtype=dt).fill_(0),
                "sizes": torch.zeros(case["formations"], case["end"] // 2 + 1, dtype=torch.int64)}
    if kind == "step":
        w = _workload(case["workload"])
        device.set_rules(w.settings)
        s, n = case["sum"], case["boards"]
        _, (l2, l4) = _layers(case, [s - 2, s - 4])
        spawned = device.expand_spawns(l2)
        boards = _unique(spawned[0], device.expand_spawns(l4)[1])
        carry = _unique(spawned[1])
        return {"case": case, "boards": _slice(boards, n, rng), "carry": _slice(carry, min(n, carry.numel() // 2), rng),
                "layer": torch.zeros(4 * n, dtype=torch.int64, device="cuda"),
                "next": torch.zeros(24 * n, dtype=torch.int64, device="cuda"),
                "carry_next": torch.zeros(24 * n, dtype=torch.int64, device="cuda")}
    w = _workload(case["workload"])
    device.set_rules(w.settings)
    s, n, p = case["sum"], case["boards"], case["precision"]
    if kind == "solve":
        _, (keys, k2, k4) = _layers(case, [s, s + 2, s + 4])
        return {"case": case, "keys": _slice(keys, n, rng), "t2": (k2, _values(k2.numel(), p, gen)),
                "t4": (k4, _values(k4.numel(), p, gen)), "win": w.formations[0].winstates, "settings": w.settings}
    # lookup: three in four boards are in the layer, each shown in one of four orientations; the others are not
    _, (keys,) = _layers(case, [s])
    at = torch.randint(0, keys.numel(), (n,), generator=gen, device="cuda")
    b = keys[at]
    b = torch.where(torch.rand(n, generator=gen, device="cuda") < 0.25, b ^ 0x10, b)
    turn = torch.randint(0, 4, (n,), generator=gen, device="cuda")
    b = torch.where((turn & 1).bool(), _transpose(b), b)
    b = torch.where((turn & 2).bool(), _mirror(b), b)
    return {"case": case, "keys": keys, "vals": _values(keys.numel(), p, gen), "boards": b}


# --------------------------------------------------------------------------- one pass
def _take(dst, at, ptr, n):
    """n values at a host pointer into dst[at:]; large blocks by torch's threads."""
    size = n * dst.element_size()
    if size < 1 << 20:
        if n:
            ctypes.memmove(dst.data_ptr() + at * dst.element_size(), ptr, size)
    else:
        src = (ctypes.c_char * size).from_address(ctypes.cast(ptr, ctypes.c_void_p).value)
        dst[at:at + n].copy_(torch.frombuffer(src, dtype=dst.dtype, count=n))


def _sort_unique(raw):
    """The distinct keys of a raw stream, ascending; the stream is sorted in place (cgb_sort)."""
    tmp = torch.empty_like(raw)
    in_tmp, passes = ctypes.c_int(), ctypes.c_int()
    _lib.check(_lib.lib().cgb_sort(raw.data_ptr(), tmp.data_ptr(), raw.numel(), ctypes.byref(in_tmp),
                                   ctypes.byref(passes)))
    return device.unique(tmp if in_tmp.value else raw)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "table":
        at = at64 = 0

        def on_table(s, kptr, vptr, n, precision):
            nonlocal at, at64
            _take(state["keys"], at, kptr, n)
            if precision == 64 and case["precision"] == 32:
                _take(state["vals64"], at64, vptr, n)
                at64 += n
            else:
                _take(state["vals"], at - at64, vptr, n)
            state["sizes"][(s - state["start"]) // 2] = n
            at += n

        device.tablebase(state["initial"], state["start"], case["end"], state["start"], state["win"],
                         precision=case["precision"], table_fn=on_table)
        return {k: state[k] for k in ("keys", "vals", "vals64", "sizes")}
    if kind == "batch":
        at = 0

        def on_formation(f, s, kptr, vptr, n, precision):
            nonlocal at
            _take(state["keys"], at, kptr, n)
            _take(state["vals"], at, vptr, n)
            state["sizes"][f, s // 2] = n
            at += n

        device.batch(state["forms"], precision=case["precision"], table_fn=on_formation)
        return {k: state[k] for k in ("keys", "vals", "sizes")}
    if kind == "step":
        layer = _sort_unique(device.expand_moves(state["boards"]))
        two, four = device.expand_spawns(layer)
        carry = _sort_unique(four)
        nxt = device.merge_unique(_sort_unique(two), state["carry"])
        for name, t in (("layer", layer), ("next", nxt), ("carry_next", carry)):
            state[name][:t.numel()].copy_(t)
        return {"layer": state["layer"], "next": state["next"], "carry_next": state["carry_next"],
                "sizes": [layer.numel(), nxt.numel(), carry.numel()]}
    if kind == "solve":
        return device.solve_layer(state["keys"], state["t2"], state["t4"], state["win"], case["precision"])
    return device.lookup_batch(state["keys"], state["vals"], state["boards"], canonicalize=True)


# --------------------------------------------------------------------------- exact values
# Boards are int64 tensors of 16 nibbles, cell 0 the most significant.
def _cells(b):
    return [(b >> (60 - 4 * c)) & 15 for c in range(16)]


def _swap(b, mask, shift):
    t = ((b >> shift) ^ b) & mask
    return b ^ t ^ (t << shift)


def _transpose(b):
    b = _swap(b, 0x0000F0F00000F0F0, 12)
    return _swap(b, 0x00000000FF00FF00, 24)


def _mirror(b):
    b = _swap(b, 0x00FF00FF00FF00FF, 8)
    return _swap(b, 0x0F0F0F0F0F0F0F0F, 4)


def _flip(b):
    b = _swap(b, 0x0000FFFF0000FFFF, 16)
    return _swap(b, 0x00000000FFFFFFFF, 32)


def _canonical(b):
    best = b ^ _SIGN
    for x in (b, _transpose(b)):
        for y in (x, _mirror(x)):
            for z in (y, _flip(y)):
                best = torch.maximum(best, z ^ _SIGN)
    return best ^ _SIGN


def _row_moves(free):
    """The left move of every row of four cells; -1 where a fixed cell would move."""
    out = []
    for row in range(65536):
        cells = [(row >> s) & 15 for s in (12, 8, 4, 0)]
        line = [c for c in cells if c]
        i = 0
        while i + 1 < len(line):
            if line[i] == line[i + 1] and line[i] < 14:
                line[i] += 1
                del line[i + 1]
            i += 1
        line += [0] * (4 - len(line))
        fixed = not free and any(c == 15 and d != 15 for c, d in zip(cells, line))
        out.append(-1 if fixed else (line[0] << 12) | (line[1] << 8) | (line[2] << 4) | line[3])
    return torch.tensor(out, dtype=torch.int64, device="cuda")


def _moves(b, rows):
    """(boards, legal) of the four moves."""
    t = _transpose(b)
    for v in (b, _mirror(b), t, _mirror(t)):
        parts = [rows[(v >> s) & 0xFFFF] for s in (48, 32, 16, 0)]
        locked = (parts[0] < 0) | (parts[1] < 0) | (parts[2] < 0) | (parts[3] < 0)
        m = (parts[0] << 48) | (parts[1] << 32) | (parts[2] << 16) | parts[3]
        yield m, ~locked & (m != v)


def _pruned(b, st):
    """The generator's prune rule: small tiles' sum, count of large tiles, third copy of a large tile."""
    cells = torch.stack(_cells(b))
    small = (cells < st.smallest_large) * (1 << cells)
    large = (cells >= st.smallest_large) & (cells < 14)
    bad = (small.sum(0) > st.stsl + 64) | (large.sum(0) > st.ltc)
    for v in range(max(st.smallest_large, 0), 14):
        bad |= (cells == v).sum(0) >= (6 if v == st.smallest_large else 3)
    return bad


def _spawned(b, value):
    out = [_canonical((b | (value << (60 - 4 * c)))[x == 0]) for c, x in enumerate(_cells(b))]
    return _unique(*out)


def _generated(initial, start, end, st):
    rows = _row_moves(st.free_formation)
    boards = torch.from_numpy(np.array(initial, np.uint64).view(np.int64)).cuda()
    carry = boards[:0]
    layers = {}
    for s in range(start, end + 1, 2):
        keep = boards[~_pruned(boards, st)] if st.prune else boards
        moved = []
        for m, legal in _moves(keep, rows):
            m = m[legal]
            moved.append(_canonical(m[~_pruned(m, st)] if st.prune else m))
        layers[s] = _unique(*moved)
        boards = _unique(_spawned(layers[s], 1), carry)
        carry = _spawned(layers[s], 2)
    return layers


def _find(keys, vals, b):
    """Float64 values of boards in a sorted layer, 0 where absent."""
    if keys.numel() == 0:
        return torch.zeros(b.shape, dtype=torch.float64, device=b.device)
    at = torch.searchsorted(keys ^ _SIGN, b ^ _SIGN).clamp_(max=keys.numel() - 1)
    return torch.where(keys[at] == b, vals[at].double(), torch.zeros((), dtype=torch.float64, device=b.device))


def _solved(keys, t2, t4, winstates, st, rows):
    out = torch.empty(keys.numel(), dtype=torch.float64, device="cuda")
    for lo in range(0, keys.numel(), 1 << 20):
        b = keys[lo:lo + (1 << 20)]
        cells = _cells(b)
        won = torch.zeros(b.shape, dtype=torch.bool, device="cuda")
        if st.nox:
            for x in cells:
                won |= x == st.nox
        else:
            for w in winstates:
                for img in _images(w):
                    mask = sum(15 << (60 - 4 * c) for c in range(16) if configs.get_tile(img, c))
                    mask, img = (v - (1 << 64) if v >= 1 << 63 else v for v in (mask, img))
                    won |= (b & mask) == img
        total = torch.zeros(b.shape, dtype=torch.float64, device="cuda")
        count = torch.zeros(b.shape, dtype=torch.float64, device="cuda")
        for c, x in enumerate(cells):
            at = torch.nonzero(x == 0).flatten()
            for value, weight, (k, v) in ((1, 0.9, t2), (2, 0.1, t4)):
                best = torch.zeros(at.shape, dtype=torch.float64, device="cuda")
                for m, legal in _moves(b[at] | (value << (60 - 4 * c)), rows):
                    p = _find(k, v, _canonical(m))
                    best = torch.where(legal, torch.maximum(best, p), best)
                total[at] += weight * best
            count[at] += 1
        out[lo:lo + b.numel()] = torch.where(won, torch.ones_like(total), total / count.clamp(min=1))
    return out


def _images(board):
    """The eight images of a board given as a Python number."""
    grid = [[configs.get_tile(board, 4 * r + q) for q in range(4)] for r in range(4)]
    for _ in range(4):
        grid = [list(r) for r in zip(*grid[::-1])]
        for g in (grid, [r[::-1] for r in grid]):
            b = 0
            for i, v in enumerate(v for r in g for v in r):
                b = configs.set_tile(b, i, v)
            yield b


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "step"):
        return None  # many small sweeps; whole numbers alone
    if kind == "table" and case["workload"] != "plain_2x4_nearwall":
        return None  # tens of millions of boards
    s = prepare(case, seed)
    if kind == "lookup":
        return _find(s["keys"], s["vals"], _canonical(s["boards"]))
    if kind == "solve":
        rows = _row_moves(s["settings"].free_formation)
        return _solved(s["keys"], s["t2"], s["t4"], s["win"], s["settings"], rows)
    st = _workload(case["workload"]).settings
    rows = _row_moves(st.free_formation)
    layers = _generated(s["initial"], s["start"], case["end"], st)
    none = (torch.zeros(0, dtype=torch.int64, device="cuda"), torch.zeros(0, dtype=torch.float64, device="cuda"))
    t2 = t4 = none
    vals, vals64 = torch.zeros(s["vals"].shape, dtype=torch.float64), torch.zeros_like(s["vals64"])
    at = at64 = 0
    for k in range(case["end"], s["start"] - 1, -2):
        v = _solved(layers[k], t2, t4, s["win"], st, rows)
        if case["precision"] == 32 and k > case["end"] - 8:
            vals64[at64:at64 + v.numel()] = v.cpu()
            at64 += v.numel()
        else:
            vals[at:at + v.numel()] = v.cpu()
            at += v.numel()
        t2, t4 = (layers[k], v), t2
    return {"keys": None, "vals": vals, "vals64": vals64, "sizes": None}
