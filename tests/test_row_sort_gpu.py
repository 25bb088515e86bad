"""Emitted rows at the edges of the row sort: one block and several tiles, rows
packed into one 64-bit key and into several, and more rows than the first emit
buffer holds.  The expected rows come from numpy (products of label classes), not
from the library."""
import numpy as np
import pytest

import matrixgraph_b200 as mg
from helpers import graph

pytestmark = pytest.mark.gpu


def bipartite(a, b, first_gid_gap=0):
    """a vertices labelled 0, each joined to all of b vertices labelled 1."""
    edges = [(i, a + j) for i in range(a) for j in range(b)]
    n = a + b + first_gid_gap
    return graph(n, edges, [0] * a + [1] * b + [2] * first_gid_gap)


@pytest.mark.parametrize("a,b", [(1, 1), (2, 4096), (64, 128), (91, 90), (3, 2731), (128, 129),
                                 (300, 301)])
def test_pairs_in_order(a, b):
    # 1, 8192 (one block exactly), 8190, 8193 (first several-tile size), 16512, 90300 rows;
    # 90300 also passes the first buffer of 65,536 rows when a cap below it is given
    dg = mg.DeviceGraph(bipartite(a, b))
    q = mg.CSRGraph.query(2, [(0, 1)], [0, 1])
    want = np.array([(i, a + j) for i in range(a) for j in range(b)], np.uint32)
    assert np.array_equal(dg.emit(q), want)
    cap = max(1, a * b // 3)
    assert np.array_equal(dg.emit(q, cap=cap), want[:cap])
    dg.free()


@pytest.mark.parametrize("leaves", [2, 4, 5])
def test_stars_packed_and_wide(leaves):
    # ids of 17 bits (70,000 vertices): 3 columns fit one key, 5 and 6 need two
    a, b = 3, {2: 60, 4: 9, 5: 7}[leaves]
    g = bipartite(a, b, first_gid_gap=70000)
    dg = mg.DeviceGraph(g)
    q = mg.CSRGraph.query(leaves + 1, [(0, 1 + x) for x in range(leaves)], [0] + [1] * leaves)
    idx = np.indices((b,) * leaves).reshape(leaves, -1).T
    idx = idx[[len(set(r)) == leaves for r in idx.tolist()]]
    want = np.concatenate([np.concatenate([np.full((len(idx), 1), c), idx + a], axis=1)
                           for c in range(a)]).astype(np.uint32)
    assert np.array_equal(dg.emit(q), want)
    dg.free()
