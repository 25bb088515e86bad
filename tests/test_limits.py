"""Limits of an enumeration call at sizes that no test puts on a device."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def limits(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("limits") / "limits")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "matrixgraph_b200", "csrc"),
                    os.path.join(ROOT, "tests", "limits_main.cpp"), "-o", exe], check=True)

    def run(*args):
        r = subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True,
                           check=True)
        return [int(x) for x in r.stdout.split()]
    return run


RUN, UNKNOWN, CHUNKED = 0, 1, 2
SEG = 1 << 30  # elements of a lane's expand launch


@pytest.mark.parametrize("t0, budget, want", [
    (0, 0, RUN), (1, 0, RUN), (SEG, 0, RUN), (SEG + 1, 0, CHUNKED), ((1 << 32) - 1, 0, CHUNKED),
    (100, 100, RUN), (101, 100, UNKNOWN), (SEG + 1, SEG, UNKNOWN), (SEG + 1, SEG + 1, CHUNKED),
])
def test_first_bucket_of_a_batch_query(limits, t0, budget, want):
    """A bucket larger than a lane's launch is counted on the chunked path: the lane
    has no kernel at level 0 that could say so, and would report 0."""
    assert limits("lane_start", t0, budget, SEG) == [want]


@pytest.mark.parametrize("epoch", [1, 2, 255])
@pytest.mark.parametrize("state", [1, 2])
@pytest.mark.parametrize("a, b", [
    (0, 0), ((1 << 42) - 1, 1), (9 * 10 ** 12, 0), ((1 << 53), (1 << 53) - 2),
    ((1 << 54) - 2, 1), ((1 << 54) - 1, 1), ((1 << 54) - 1, 1 << 42), (1 << 61, 1 << 42),
])
def test_look_back_words(limits, epoch, state, a, b):
    """Element sums pass 2^42 unharmed and stop at the largest value, in words that
    keep their epoch and state."""
    most = (1 << 54) - 1
    assert limits("look_back", epoch, state, a, b) == [epoch, state, min(a + b, most), most, 255]


MIN, TRY = 1 << 16, 1 << 22
GIB = 1 << 30


@pytest.mark.parametrize("cap, limit, row, want", [
    (0, GIB, 33, MIN), (1, GIB, 33, MIN), (MIN, GIB, 33, MIN), (MIN + 1, GIB, 33, MIN + 1),
    (TRY, GIB, 33, TRY), (TRY + 1, GIB, 33, TRY + 1), (5 * 10 ** 6, GIB, 33, 5 * 10 ** 6),
    (GIB // 33, GIB, 33, GIB // 33), (GIB // 33 + 1, GIB, 33, 0), ((1 << 31) - 1, GIB, 33, 0),
    (1 << 31, GIB, 0, 0), ((1 << 64) - 1, GIB, 33, 0), (10, MIN * 33 - 1, 33, 0),
])
def test_room_for_a_callers_buffer(limits, cap, limit, row, want):
    """The whole buffer or a count first: never an attempt at part of it."""
    assert limits("emit_room", 1, cap, 0, limit, 0, row) == [want]


KEEP = 1 << 28


@pytest.mark.parametrize("entries, limit, held, want", [
    (0, KEEP, 0, MIN), (110_000, KEEP, 0, 1 << 19), (MIN // 4, KEEP, 0, MIN),
    (MIN // 4 + 1, KEEP, 0, 2 * MIN), (1 << 30, KEEP, 0, TRY), (1 << 30, 33 << 20, 0, 1 << 20),
    (1 << 30, 33 * MIN - 1, 0, 0),
    # what the graph holds already is used, however small the graph
    (0, KEEP, 33 * MIN * 8, MIN * 8), (0, KEEP, 33 * MIN * 8 - 1, MIN * 4), (0, 0, 33 * TRY, TRY),
])
def test_room_for_any_number_of_rows(limits, entries, limit, held, want):
    assert limits("emit_room", 0, (1 << 64) - 1, entries, limit, held, 33) == [want]


def test_room_of_a_large_held_block(limits):
    """A block that is there serves a caller's buffer beyond the limit, too."""
    assert limits("emit_room", 1, 10 ** 7, 0, KEEP, 33 * 10 ** 7, 33) == [10 ** 7]
    assert limits("emit_room", 1, 10 ** 7, 0, KEEP, 33 * 10 ** 7 - 1, 33) == [0]


# rows of 25, 29, 33 bytes at levels 1, 2, 3; a call of 4 vertices uses the three
@pytest.mark.parametrize("cap, budget, rows, want", [
    (1000, 87_000, [], []),
    (1000, 87_000, [4, 1000, 1000, 1000], []),
    (1000, 87_000, [4, 1001], [1]),              # level 1 as it is, 2 and 3 grown to cap
    (1000, 90_000, [4, 1001], []),
    (1000, 87_000, [4, 500, 3000, 10], [2]),     # within the budget alone, not once grown
    (1000, 87_000, [4, 500, 500, 500, 1], [4]),  # a level that this call does not use
    (1000, 87_000, [4, 2000, 500, 2000, 0, 7], [1, 3, 5]),
    (1, 87, [1 << 20], []),                      # level 0 is the call's queries
])
def test_tables_of_earlier_calls_under_a_budget(limits, cap, budget, rows, want):
    got = limits("tables", 4, cap, budget, *rows)
    assert got == want
    size = {1: 25, 2: 29, 3: 33, 4: 37, 5: 41}
    left = {level: n for level, n in enumerate(rows) if level and n and level not in got}
    held = {level: max(left.get(level, 0), cap) for level in (1, 2, 3)}
    held.update({level: n for level, n in left.items() if level > 3})
    assert sum(n * size[level] for level, n in held.items()) <= budget
