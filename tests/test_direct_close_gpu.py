"""Candidates closed where they are found (a last position, a pendant tail),
against the oracle: own and earlier anchors, up to two further constraints, zero
to three open look-ups, empty slices, self-loops, look-ups in hub bitmaps and in
slices; and positions that intersect two or three lists."""
import itertools

import numpy as np
import pytest

import matrixgraph_b200 as mg
from helpers import graph, oracle_count, random_graph

pytestmark = pytest.mark.gpu

SHAPES = {
    "path4": [(0, 1), (1, 2), (2, 3)],
    "path5": [(0, 1), (1, 2), (2, 3), (3, 4)],
    "fork": [(0, 1), (1, 2), (1, 3), (3, 4)],
    "star4": [(0, 1), (0, 2), (0, 3), (3, 4)],
    # the position that closes has a further constraint, or two
    "triangle-tail1": [(0, 1), (1, 2), (0, 2), (2, 3)],
    "triangle-tail2": [(0, 1), (1, 2), (0, 2), (2, 3), (3, 4)],
    "square-tail2": [(0, 1), (1, 2), (2, 3), (0, 3), (1, 4), (4, 5)],
    "clique-tail1": [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3), (1, 4)],
    # two and three lists intersected, at a last position and before one
    "square": [(0, 1), (1, 2), (2, 3), (0, 3)],
    "clique": [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)],
    "clique-roof": [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3), (2, 4), (3, 4)],
}


@pytest.mark.parametrize("hub_bytes", [0, 1 << 24])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_few_labels(shape, hub_bytes):
    rng = np.random.default_rng([len(shape), hub_bytes])
    edges = SHAPES[shape]
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
        for qi in rng.choice(len(orders), min(8, len(orders)), replace=False):
            order = orders[int(qi)]
            q = mg.CSRGraph.query(k, edges, rng.integers(0, n_labels, k))
            want = oracle_count(g, q, order=order)
            got, st = dg.count(q, given_order=order, stats=True)
            assert got == want["count"], (shape, order, q.array("labels").tolist())
            assert st["level_rows"] == want["level_rows"]
            assert st["balg_bytes"] == want["balg"]
            assert st["balg_count_bytes"] == want["balg_count"]
        dg.free()
