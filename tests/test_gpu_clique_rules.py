"""4-cliques on graphs with few triangles: vertices that the edges' supports rule out,
and graphs of short lists, which are merged.  Whole numbers: equality with closed
forms or the oracle."""
from math import comb

import numpy as np
import pytest

import fsgc
import oracle
from helpers import EXTRA

pytestmark = pytest.mark.gpu
CLIQUE, TAILS = EXTRA["4clique"], EXTRA["tailed_4clique_2"]


@pytest.mark.parametrize("c", [3, 4, 5, 8, 9, 10, 12])
def test_rings_of_cliques(ctx, c):
    """Out-degrees on both sides of the rule; single and packed, wrapping and exact."""
    k = 50
    i, j = np.triu_indices(c, 1)
    pairs = np.concatenate([np.stack([i, j], 1) + c * t for t in range(k)] +
                           [np.stack([np.arange(k) * c, (np.arange(1, k + 1) % k) * c + 1], 1)])
    g = fsgc.csr_from_edges(c * k, pairs)
    d = g.degrees()
    gid, pid = ctx.upload(g), ctx.upload_packed([g, fsgc.gen_rmat(8, 8, seed=2), g])
    try:
        want = {CLIQUE[0]: k * comb(c, 4)}
        # every clique of a vertex, times the pairs of its other neighbours
        want[TAILS[0]] = sum(comb(c - 1, 3) * comb(max(0, int(x) - 3), 2) for x in d)
        for p in (CLIQUE, TAILS):
            mo = fsgc.preprocess(*p)
            assert ctx.count(gid, mo).raw_total == want[p[0]]
            assert ctx.count_exact(gid, mo).raw_total == want[p[0]]
            packed = ctx.count_packed(pid, mo)
            assert [packed[0].raw_total, packed[2].raw_total] == [want[p[0]]] * 2
    finally:
        ctx.release(gid)
        ctx.release(pid)


def late_clique(extras, at_least):
    """A vertex whose `extras` first out-edges are in no triangle and whose last three
    close a 4-clique; every other vertex has `at_least` neighbours or is a leaf."""
    a, xyz = 0, [extras + 1, extras + 2, extras + 3]
    pairs = [(a, b) for b in range(1, extras + 4)]
    pairs += [(xyz[0], xyz[1]), (xyz[0], xyz[2]), (xyz[1], xyz[2])]
    v = extras + 4
    for b in range(1, extras + 4):
        pairs += [(b, v + t) for t in range(at_least)]
        v += at_least
    return fsgc.csr_from_edges(v, pairs)


@pytest.mark.parametrize("extras", [7, 28, 29, 30, 31, 125, 126, 127, 128, 260])
def test_cliques_at_the_end_of_a_list(ctx, extras):
    g = late_clique(extras, extras + 6)
    gid = ctx.upload(g)
    try:
        for p in (CLIQUE, TAILS):
            mo = fsgc.preprocess(*p)
            assert ctx.count(gid, mo).raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"]
        assert ctx.count(gid, fsgc.preprocess(*CLIQUE)).raw_total == 1
    finally:
        ctx.release(gid)


@pytest.mark.parametrize("g", [fsgc.gen_er(3000, 9000, 1), fsgc.gen_er(2000, 30_000, 2), fsgc.gen_er(400, 16_000, 3),
                               fsgc.gen_chung_lu(5000, 6.0, 2.4, 4)], ids=["sparse", "er", "dense", "hubs"])
def test_few_and_many_triangles_against_the_oracle(ctx, g):
    gid = ctx.upload(g)
    try:
        for p in (CLIQUE, TAILS):
            mo = fsgc.preprocess(*p)
            assert ctx.count(gid, mo).raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"]
    finally:
        ctx.release(gid)
