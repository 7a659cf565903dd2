"""The order of the parts that thread blocks of one launch share (csrc/split_schedule.cuh, built here with the host compiler): nobody may wait for a
block that can only start after it, however few blocks the launch gets at a time."""
import ctypes
import random
import subprocess
from pathlib import Path

import pytest

from tests.test_streamk_protocol import SHAPES, SK_BN, TG_BK, owner_last, segments

CSRC = Path(__file__).resolve().parents[1] / "mistral_inference_b200" / "csrc"
SOURCE = """
#include "split_schedule.cuh"
extern "C" void plan(long long pairs, int num_k, int units, int max_parts, int* out) {
  const mb200::CutPlan c = mb200::cut_plan(pairs, num_k, units, max_parts);
  out[0] = c.cut_pairs; out[1] = c.cut;
}
extern "C" void item(int s, int cut, int cut_pairs, int* out) {
  const mb200::CutItem i = mb200::cut_item(s, cut, cut_pairs);
  out[0] = i.part; out[1] = i.slot;
}
extern "C" int range(int block, int grid) { return mb200::streamk_range(block, grid); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("schedule")
    (d / "s.cc").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), "-o", str(d / "s.so"), str(d / "s.cc")], check=True)
    handle = ctypes.CDLL(str(d / "s.so"))
    handle.plan.argtypes = [ctypes.c_longlong] + [ctypes.c_int] * 3 + [ctypes.POINTER(ctypes.c_int)]

    def call(f, *a):
        out = (ctypes.c_int * 2)()
        f(*a, out)
        return tuple(out)

    return type("Lib", (), dict(plan=staticmethod(lambda *a: call(handle.plan, *a)), item=staticmethod(lambda *a: call(handle.item, *a)), range=staticmethod(handle.range)))


def run_blocks(steps, resident, r):
    """Blocks start in the order of their index while fewer than `resident` are on the chip and leave at their end.  steps[b]: what block b does,
    ("post", x) or ("wait", x).  A wait that can never end fails."""
    posted, on, nxt = set(), [], 0
    pos = [0] * len(steps)
    while on or nxt < len(steps):
        while len(on) < resident and nxt < len(steps):
            on.append(nxt)
            nxt += 1
        ready = [b for b in on if pos[b] == len(steps[b]) or steps[b][pos[b]][0] == "post" or steps[b][pos[b]][1] in posted]
        assert ready, f"{len(on)} blocks wait for parts that cannot start"
        b = r.choice(ready)
        if pos[b] == len(steps[b]):
            on.remove(b)
            continue
        kind, x = steps[b][pos[b]]
        if kind == "post":
            posted.add(x)
        pos[b] += 1
    return posted


@pytest.mark.parametrize("units", [74, 66, 5])
def test_owners_of_cut_pairs_wait_for_earlier_clusters_only(lib, units):
    r = random.Random(units)
    seen = set()
    for _ in range(60):
        pairs, num_k = r.randint(1, 6 * units), r.choice([4, 8, 17, 32, 64, 224])
        cut_pairs, cut = lib.plan(pairs, num_k, units, 56)
        if cut_pairs == 0:
            assert cut == 1
            continue
        seen.add(cut)
        assert cut_pairs == pairs % units and 2 <= cut <= 4 and cut * cut_pairs <= units and num_k >= 8 * cut and (cut - 1) * cut_pairs <= 56
        items = [lib.item(s, cut, cut_pairs) for s in range(cut * cut_pairs)]
        assert sorted(items) == [(p, s) for p in range(cut) for s in range(cut_pairs)], "every part of every pair once"
        steps = [[("post", it)] if it[0] else [("wait", (o, it[1])) for o in range(1, cut)] for it in items]
        for resident in (1, 2, units // 2, units):
            run_blocks(steps, max(resident, 1), r)
    assert seen >= ({2, 3, 4} if units > 5 else {2})


@pytest.mark.parametrize("G", [148, 37, 3])
def test_streamk_owners_wait_for_earlier_blocks_only(lib, G):
    """The ranges and roles are those of test_streamk_protocol; here their blocks start one after the other."""
    r = random.Random(G)
    for N, K in SHAPES[::4]:
        num_k = K // TG_BK
        total = N // SK_BN * num_k
        grid = min(G, total)
        steps = []
        for block in range(grid):
            c, mine = lib.range(block, grid), []
            for tile, kb0, kb1 in segments(total, num_k, grid, c):
                if kb0 != 0:
                    mine.append(("post", c))
                elif kb1 != num_k:
                    mine += [("wait", o) for o in range(c + 1, owner_last(total, num_k, grid, c, tile) + 1)]
            steps.append(mine)
        assert sorted(lib.range(b, grid) for b in range(grid)) == list(range(grid))
        for resident in (1, grid // 2 + 1, grid):
            run_blocks(steps, resident, r)
