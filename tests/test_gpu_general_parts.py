"""General cores on the bit matrix of sparse graphs, where the lists are too short to be
split over many tasks: every number of parts, against the oracle."""
import numpy as np
import pytest

import fsgc
import oracle
from helpers import EXTRA

pytestmark = pytest.mark.gpu


def path(n):
    return fsgc.csr_from_edges(n, np.stack([np.arange(n - 1), np.arange(1, n)], 1))


def ring_of_squares(k):
    """Squares sharing corners: degrees 2 and 4."""
    pairs = []
    for i in range(k):
        a, b, c, d = 3 * i, 3 * i + 1, 3 * i + 2, 3 * ((i + 1) % k)
        pairs += [(a, b), (b, d), (d, c), (c, a)]
    return fsgc.csr_from_edges(3 * k, pairs)


GRAPHS = {
    "path": lambda: path(300),
    "squares": lambda: ring_of_squares(60),
    "sparse": lambda: fsgc.gen_er(500, 600, 1),
    "five a vertex": lambda: fsgc.gen_er(300, 750, 2),
    "ten a vertex": lambda: fsgc.gen_er(60, 300, 3),
    "hub": lambda: fsgc.csr_from_edges(80, [(0, i) for i in range(1, 40)] + [(i, i + 1) for i in range(1, 79)]),
}
PATTERNS = [EXTRA["5cycle"], EXTRA["5cycle_chord_fringe"], (6, [(0, 1), (1, 2), (2, 3), (3, 0), (0, 4), (2, 5)]),
            (8, [(0, 1), (1, 2), (2, 3), (0, 4), (0, 5), (3, 6), (1, 7)])]


@pytest.mark.parametrize("name", list(GRAPHS))
def test_sparse_graphs(ctx, name):
    g = GRAPHS[name]()
    gid = ctx.upload(g)
    try:
        for n, e in PATTERNS:
            mo = fsgc.preprocess(n, e)
            assert ctx.count(gid, mo).raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"], (n, e)
    finally:
        ctx.release(gid)
