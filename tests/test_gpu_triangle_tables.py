"""Triangle core by out-neighbour tables: the vertex sizes at which the kernels
change over (rows in shared memory, in slabs, in the arena; narrow and wide
blocks; a hub with few out-neighbours), against closed forms on cliques with
pendant leaves and the oracle on a hub graph.  Whole numbers: equality."""
from math import comb

import pytest

import fsgc
import oracle
from helpers import EXTRA, WORKLOAD

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


def clique_with_leaves(c, leaves):
    """K_c, every clique vertex with `leaves` pendant neighbours of its own."""
    pairs = [(i, j) for i in range(c) for j in range(i + 1, c)]
    v = c
    for i in range(c):
        pairs += [(i, v + t) for t in range(leaves)]
        v += leaves
    return fsgc.csr_from_edges(v, pairs)


@pytest.mark.parametrize("c,leaves", [(33, 0), (40, 700), (300, 3000), (300, 2), (900, 0)])
def test_cliques_with_leaves(ctx, c, leaves):
    """(33, 0): just past a warp's table; (40, 700): narrow rows; (300, 3000):
    rows beyond shared memory; (300, 2): the wide table; (900, 0): 4-clique rows
    in slabs."""
    gid = ctx.upload(clique_with_leaves(c, leaves))
    try:
        d = c - 1 + leaves
        assert ctx.count(gid, fsgc.preprocess(*EXTRA["4clique"])).raw_total == comb(c, 4)
        tailed = fsgc.preprocess(*EXTRA["tailed_4clique_2"])
        assert ctx.count(gid, tailed).raw_total == (comb(c, 4) * 4 * comb(d - 3, 2)) & M64
        if c > 400:
            return
        # a fringe on all three, then one on each: the three choose disjointly
        # from c - 4 vertices they share and their own leaves
        r, n = c - 4, c - 4 + leaves
        want = comb(c, 3) * (c - 3) * (n ** 3 - 3 * n * r + 2 * r)
        mo = fsgc.preprocess(*WORKLOAD["4clique_3_distinct"])
        assert ctx.count(gid, mo).raw_total == want & M64
        assert ctx.count_exact(gid, mo).raw_total == want
    finally:
        ctx.release(gid)


@pytest.mark.parametrize("leaves", [300, 4200])
def test_hubs_with_few_out_neighbours(ctx, leaves):
    """Three adjacent hubs over the same leaves: the lowest has two
    out-neighbours and more lists than one warp, or a narrow block, reads."""
    pairs = [(0, 1), (0, 2), (1, 2)] + [(h, 3 + t) for t in range(leaves) for h in range(3)] + [(3, 4), (4, 5)]
    g = fsgc.csr_from_edges(leaves + 3, pairs)
    gid = ctx.upload(g)
    try:
        for name in ("4clique", "tailed_4clique_2", "triangle_mixed"):
            mo = fsgc.preprocess(*EXTRA[name])
            o = oracle.count(g.nindex, g.nlist, mo.to_bytes())
            assert ctx.count(gid, mo).raw_total == o["raw"], name
    finally:
        ctx.release(gid)
