"""What a launch keeps in shared memory beside its points (a table of folded entries, the points' reciprocals;
pacuda_b200/csrc/shapes.h): the points per block that the caller or the tuner chose, and a point of every plan, fit
wherever they fit without either, and with room for all of it nothing is left out."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HARNESS = os.path.join(os.path.dirname(__file__), "harness")


@pytest.fixture(scope="module")
def lib():
    subprocess.run(["make", "-s", "-C", HARNESS, "libshapes_harness.so"], check=True)
    return C.CDLL(os.path.join(HARNESS, "libshapes_harness.so"))


def shapes(lib, plans, room, spread=False, threads=512):
    sizes = np.array(plans, dtype=np.uint64).reshape(-1, 5)
    out, table = np.zeros((len(sizes), 2), np.uint32), C.c_uint64(0)
    ok = lib.shapes(C.c_void_p(sizes.ctypes.data), len(sizes), threads, C.c_uint64(room), int(spread), C.byref(table),
                    C.c_void_p(out.ctypes.data))
    return (table.value, out) if ok else None


def test_launches_around_the_limits(lib):
    rng = np.random.default_rng(4)
    seen = set()
    for _ in range(20000):
        n = int(rng.integers(1, 5))
        room = int(rng.choice([232400, 115664, 57320, 13300]))
        plans = []
        for _ in range(n):
            points = int(rng.choice([1, 2, 3, 4, 5, 6, 8, 10, 16, 32]))
            # a point's bytes near the limit for this count, in 16-byte steps
            bare = max(16, room // points // 16 * 16 - 16 * int(rng.integers(-4, 24)))
            plans.append((bare + 16 * int(rng.integers(0, 15)), bare, 16 * int(rng.integers(0, 257)), points,
                          int(rng.integers(0, 2))))
        spread = bool(rng.integers(0, 8) == 0)
        got = shapes(lib, plans, room, spread)
        assert (got is not None) == all(p[1] <= room for p in plans)
        if got is None:
            continue
        table, out = got
        assert table in (0, max(p[2] for p in plans))
        seen.add((table > 0, bool(out[:, 1].all())))
        for (kept, bare, _, points, chosen), (per, keep) in zip(plans, out):
            assert 1 <= per <= 32 and table + per * (kept if keep else bare) <= room
            if spread:
                assert per == 1
            elif chosen and points * bare <= room:
                assert per == points
            assert keep == (table + per * kept <= room)
        if all(max(p[2] for p in plans) + (1 if spread else p[3]) * p[0] <= room for p in plans):
            assert table == max(p[2] for p in plans) and out[:, 1].all()
            assert spread or [int(p[3]) for p in plans] == out[:, 0].tolist()
    assert len(seen) == 4


def test_default_points(lib):
    # of the counts that fit, the one that leaves the fewest threads of a warp idle, the larger on ties
    assert shapes(lib, [(11440, 11360, 144, 0, 0)], 232400)[1].tolist() == [[16, 1]]
    assert shapes(lib, [(45000, 44900, 144, 0, 0)], 232400)[1].tolist() == [[4, 1]]
    assert shapes(lib, [(232390, 232300, 144, 0, 0)], 232400) [0] == 0  # a point, and no room for the table
    assert shapes(lib, [(232500, 232400, 144, 0, 0)], 232400)[1].tolist() == [[1, 0]]
