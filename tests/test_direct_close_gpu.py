"""Candidates closed where they are found (a last position or a pendant tail
hanging off a position with one backward neighbour), against the oracle: own
and earlier anchors, zero to three open look-ups, empty slices, self-loops,
look-ups in hub bitmaps and in slices."""
import itertools

import numpy as np
import pytest

import matrixgraph_b200 as mg
from helpers import graph, oracle_count, random_graph

pytestmark = pytest.mark.gpu

TREES = {
    "path4": [(0, 1), (1, 2), (2, 3)],
    "path5": [(0, 1), (1, 2), (2, 3), (3, 4)],
    "fork": [(0, 1), (1, 2), (1, 3), (3, 4)],
    "star4": [(0, 1), (0, 2), (0, 3), (3, 4)],
}


@pytest.mark.parametrize("hub_bytes", [0, 1 << 24])
@pytest.mark.parametrize("shape", list(TREES))
def test_trees_of_few_labels(shape, hub_bytes):
    rng = np.random.default_rng([len(shape), hub_bytes])
    edges = TREES[shape]
    k = max(max(e) for e in edges) + 1
    for loops, n_labels in ((False, 1), (False, 2), (True, 2), (False, 3)):
        e, labels = random_graph(rng, 24, 0.18, n_labels)
        if loops:
            e = e + [(v, v) for v in range(0, 24, 3)]
        g = graph(24, e, labels)
        dg = mg.DeviceGraph(g, hub_bytes=hub_bytes, hub_min_degree=1)
        orders = [o for o in itertools.permutations(range(k))
                  if all(any((a, b) in edges or (b, a) in edges for b in o[:i])
                         for i, a in enumerate(o) if i)]
        for qi in rng.choice(len(orders), 6, replace=False):
            order = orders[int(qi)]
            q = mg.CSRGraph.query(k, edges, rng.integers(0, n_labels, k))
            want = oracle_count(g, q, order=order)
            got, st = dg.count(q, given_order=order, stats=True)
            assert got == want["count"], (shape, order, q.array("labels").tolist())
            assert st["level_rows"] == want["level_rows"]
            assert st["balg_bytes"] == want["balg"]
            assert st["balg_count_bytes"] == want["balg_count"]
        dg.free()
