"""The walk over the level tables where it stops and goes on: levels larger than
their table, more blocks than tiles, and the limits of a call, against the oracle."""
import itertools

import numpy as np
import pytest

import matrixgraph_b200 as mg
from matrixgraph_b200 import _lib as L
from helpers import oracle_count, oracle_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dense():
    """R-MAT scale 12 with four labels: a 4-cycle has 11,119 rows at level 2, whose
    candidate elements pass a table of 2^17 rows."""
    g = mg.rmat(12, n_labels=4)
    dg = mg.DeviceGraph(g)
    yield g, dg
    dg.free()


@pytest.mark.parametrize("chunk_rows", [1000, 1 << 16, 1 << 17])
@pytest.mark.parametrize("shape", ["4-cycle", "4-clique"])
def test_stopped_levels_are_walked_again_alike(dense, shape, chunk_rows):
    """A level that passes its table stops the chain from within the launch that
    measures it, while most of that launch's blocks have no tile: every repetition
    walks the same rows."""
    g, dg = dense
    q = mg.query_walk(g, shape, seed=3)
    want = oracle_count(g, q, threads=4)
    for _ in range(1 if chunk_rows < 4096 else 40):
        got, st = dg.count(q, stats=True, chunk_rows=chunk_rows)
        assert got == want["count"]
        assert st["level_rows"] == want["level_rows"]
        assert st["balg_bytes"] == want["balg"]


def test_chained_levels_read_what_the_level_before_wrote(dense):
    """Calls of many levels back to back, whose launches overlap and share one table
    of tile rows: three queries of other sizes in turn, each the same every time."""
    g, dg = dense
    qs = [mg.query_walk(g, s, seed=7) for s in ("4-cycle", "4-clique", "tailed-triangle")]
    want = [oracle_count(g, q, threads=4) for q in qs]
    for q in qs:  # tables grow to what the queries need
        dg.count(q, no_tail=1)
    for _ in range(40):
        for q, w in zip(qs, want):
            got, st = dg.count(q, stats=True, no_tail=1)
            assert got == w["count"] and st["level_rows"] == w["level_rows"]


def test_batch_after_lanes_that_did_not_fit(dense):
    """Lane tables for 2^31 rows (over 400 GB) are refused as often as they are asked
    for, and leave nothing behind that a later batch would use."""
    g, dg = dense
    qs = [mg.query_walk(g, "4-clique", seed=s) for s in range(3)]
    want = [oracle_count(g, q, threads=4)["count"] for q in qs]
    for _ in range(2):
        with pytest.raises(L.MGError) as e:
            dg.batch_count(qs, chunk_rows=1 << 31, lanes=2)
        assert e.value.code == L.MG_E_OOM
    assert dg.batch_count(qs, lanes=2).tolist() == want
    assert dg.batch_count(qs * 40, lanes=2).tolist() == want * 40
    assert dg.batch_count(qs, lanes=2).tolist() == want


def test_level_of_more_than_2_42_elements_meets_the_budget():
    """A second vertex that is not joined to the first: 2.2M rows of 2.2M candidates
    each, refused by the work budget in a single call and reported as unknown in a
    batch, whose other queries are counted."""
    n = 2_200_000
    v = np.arange(n, dtype=np.uint32)
    g = mg.CSRGraph.from_edges(n, v, np.roll(v, -1), np.zeros(n, np.uint32), symmetrize=True)
    dg = mg.DeviceGraph(g)
    q = mg.CSRGraph.query(3, [(0, 1), (1, 2)], [0, 0, 0])
    with pytest.raises(L.MGError) as e:
        dg.count(q, given_order=[0, 2, 1], max_elements=1 << 30)
    assert e.value.code == L.MG_E_LIMIT
    counts, _, _ = dg.batch_count_orders([q, q], [[0, 2, 1], [1, 0, 2]], max_elements=1 << 30)
    assert counts.tolist() == [2 ** 64 - 1, 2 * n]
    assert dg.count(q) == 2 * n
    dg.free()


def test_more_work_scans_than_epochs(dense):
    """Hundreds of chunks in one call: the look-back words are cleared when their
    epochs run out."""
    g, dg = dense
    q = mg.query_walk(g, "4-cycle", seed=3)
    want = oracle_count(g, q, threads=4)
    got, st = dg.count(q, stats=True, chunk_rows=1500)
    assert st["chunks"] > 600
    assert got == want["count"] and st["level_rows"] == want["level_rows"]


def test_emit_falls_back_only_when_its_buffer_is_full(dense):
    """An emit whose matches pass its buffer counts and emits again, and its launches
    say so; one that its budget refuses is refused at once and counted as nothing."""
    g, dg = dense
    q = mg.query_walk(g, "4-clique", seed=7)
    want = oracle_rows(g, q)
    assert len(want) > 1 << 16  # rows that an attempt has room for at least
    for _ in range(2):  # (the level tables have grown at the second call)
        counted = dg.count(q, stats=True)[1]["launches"]
        dg.emit(q, cap=len(want))
    rows, n, once = dg.emit(q, cap=len(want), stats=True)
    assert n == len(want) and np.array_equal(rows, want)
    rows, n, again = dg.emit(q, cap=10, stats=True)
    assert n == len(want) and np.array_equal(rows, want[:10])
    assert again["launches"] >= once["launches"] + counted
    with pytest.raises(L.MGError) as e:
        dg.emit(q, max_elements=1000)
    assert e.value.code == L.MG_E_LIMIT
    assert np.array_equal(dg.emit(q), want)


def test_emit_of_more_than_2_22_rows_is_one_enumeration():
    """5 million edges of a ring of chords, written into a buffer of just their size:
    as many launches as levels, and the rows are the edges."""
    n, chords = 50_000, 50
    v = np.repeat(np.arange(n, dtype=np.uint32), chords)
    w = (v + np.tile(np.arange(1, chords + 1, dtype=np.uint32), n)) % n
    g = mg.CSRGraph.from_edges(n, v, w, np.zeros(n, np.uint32), symmetrize=True)
    dg = mg.DeviceGraph(g)
    q = mg.CSRGraph.query(2, [(0, 1)], [0, 0])
    total = 2 * n * chords
    assert total > 1 << 22
    dg.emit(q, cap=total)  # (the level tables have grown at the second call)
    rows, got, st = dg.emit(q, cap=total, stats=True)
    assert got == total and st["launches"] <= 4
    both = np.concatenate([np.stack([v, w], 1), np.stack([w, v], 1)]).astype(np.uint32)
    assert np.array_equal(rows, both[np.lexsort((both[:, 1], both[:, 0]))])
    dg.free()


def test_small_graph_keeps_a_small_emit_block():
    """The first emit of a graph of some ten thousand edges does not take room for
    millions of rows."""
    torch = pytest.importorskip("torch")
    g = mg.chung_lu(2000, avg_deg=6, n_labels=4)
    dg = mg.DeviceGraph(g)
    q = mg.CSRGraph.query(4, [(0, 1), (1, 2), (2, 3), (3, 0)], [0, 1, 0, 1])
    n = dg.count(q)  # the level tables
    before = torch.cuda.mem_get_info()[0]
    assert np.array_equal(dg.emit(q), oracle_rows(g, q)) and n == len(dg.emit(q))
    assert before - torch.cuda.mem_get_info()[0] <= 32 << 20
    dg.free()


def test_memory_budget_covers_tables_of_earlier_calls():
    """A call without a budget leaves a large table at level 1; one with a budget of
    56 MiB, whose deeper levels grow as far as they may, stays within it."""
    torch = pytest.importorskip("torch")
    n = 1 << 21
    v = np.arange(n, dtype=np.uint32)
    g = mg.CSRGraph.from_edges(n, np.tile(v, 3), np.concatenate([np.roll(v, -s) for s in (1, 2, 3)]),
                               np.zeros(n, np.uint32), symmetrize=True)
    dg = mg.DeviceGraph(g, hub_bytes=0)
    first = torch.cuda.mem_get_info()[0]
    path = mg.CSRGraph.query(3, [(0, 1), (1, 2)], [0] * 3)
    cycle = mg.CSRGraph.query(4, [(0, 1), (1, 2), (2, 3), (3, 0)], [0] * 4)
    # every vertex has neighbours at these distances
    steps = (-3, -2, -1, 1, 2, 3)
    closed = [(a, a + b, a + b + c) for a in steps for b in steps for c in steps
              if len({0, a, a + b, a + b + c}) == 4 and -(a + b + c) in steps]
    # (the path's last position is closed in place: one table, of 2^21 rows)
    assert dg.count(path, no_tail=1, chunk_rows=1 << 21) == n * 6 * 5
    budget = 56 << 20
    assert dg.count(cycle, mem_budget_bytes=budget) == n * len(closed)
    held = first - torch.cuda.mem_get_info()[0]
    assert held <= budget + (16 << 20)  # and the scratch that is not tables
    dg.free()


@pytest.mark.parametrize("k", [4, 5])
def test_tail_sums_in_place_without_memory_for_its_table(k):
    """A pendant tail whose table (48 MiB here) does not fit the free memory is summed
    where it is closed; with memory, the same call takes the table."""
    torch = pytest.importorskip("torch")
    # A ring with chords; every fourth vertex carries the label of the path's end.
    path = mg.CSRGraph.query(k, [(i, i + 1) for i in range(k - 1)], [0] * (k - 1) + [1])
    per_4 = 0
    for start in range(4):
        for steps in itertools.product((-2, -1, 1, 2), repeat=k - 1):
            at = np.cumsum((start,) + steps)
            per_4 += len(set(at.tolist())) == k and \
                (at % 4 == 3).tolist() == [False] * (k - 1) + [True]

    def ring(n):
        v = np.arange(n, dtype=np.uint32)
        g = mg.CSRGraph.from_edges(n, np.tile(v, 2), np.concatenate([np.roll(v, -1), np.roll(v, -2)]),
                                   (v % 4 == 3).astype(np.uint32), symmetrize=True)
        return g, mg.DeviceGraph(g, hub_bytes=0)

    g, dg = ring(1000)
    assert dg.count(path) == 250 * per_4 > 0  # (its kernels are loaded)
    dg.free()
    n = 1 << 22
    table = 16 * (n - n // 4)
    g, dg = ring(n)
    assert dg.count(path, no_tail=1) == n // 4 * per_4  # the level tables
    torch.cuda.synchronize()
    filler = [torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8,
                          device="cuda")]
    try:  # what the driver keeps back for allocations, too
        while True:
            filler.append(torch.empty(16 << 20, dtype=torch.uint8, device="cuda"))
    except torch.OutOfMemoryError:
        pass
    del filler[-1:]
    torch.cuda.empty_cache()  # 16 MiB and less than a chunk are left
    assert dg.count(path) == n // 4 * per_4
    del filler
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    assert dg.count(path) == n // 4 * per_4
    assert free - torch.cuda.mem_get_info()[0] >= table  # the table is there now
    dg.free()
