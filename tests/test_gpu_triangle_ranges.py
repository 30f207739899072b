"""Triangle core at out-degrees of 2,049 and more: ids and degrees read from memory
instead of shared memory (beyond 2,048), 4-clique rows in slabs down to one word
(6,000), and the kernel that merges lists (beyond 8,192), on two complete sides with a
few edges inside each, which have few triangles; a clique of 2,237; and supports in
rank order on packed graphs.  Closed forms, themselves checked against the oracle."""
from math import comb

import numpy as np
import pytest

import fsgc
import oracle
from helpers import EXTRA, WORKLOAD

M64 = (1 << 64) - 1
PATTERNS = {
    "4clique": EXTRA["4clique"],
    "tails": EXTRA["tailed_4clique_2"],
    "on all three, one each": WORKLOAD["4clique_3_distinct"],
    "one each": (6, [(0, 1), (0, 2), (1, 2), (0, 3), (1, 4), (2, 5)]),
}


def two_sides(p, a, b):
    """K(p, p) with `a` disjoint edges inside one side and `b` inside the other."""
    partner = {}
    for first, pairs in ((0, a), (p, b)):
        for v in range(first, first + 2 * pairs, 2):
            partner[v], partner[v + 1] = v + 1, v
    off = np.zeros(2 * p + 1, np.int64)
    adj = []
    for v in range(2 * p):
        row = np.arange(p, 2 * p, dtype=np.int32) if v < p else np.arange(p, dtype=np.int32)
        if v in partner:
            row = np.sort(np.append(row, np.int32(partner[v])))
        adj.append(row)
        off[v + 1] = off[v] + len(row)
    return fsgc.Graph(off, np.concatenate(adj))


def totals(p, a, b):
    """Raw totals of PATTERNS on two_sides(p, a, b)."""
    cliques = a * b  # an edge of either side; each vertex has degree p + 1

    def one_each(edge):
        """Triangle (x, x', y), y on an inside edge of its own (edge = 1) or not:
        disjoint choices from N(x), N(x'), N(y) without the triangle."""
        x, y = p - 1, p - 2 + edge  # N(x) and N(x') coincide, N(y) meets them in its partner
        return x * x * y - x * y - 2 * x * edge + 2 * edge

    both = a * (2 * b * one_each(1) + (p - 2 * b) * one_each(0)) + b * (2 * a * one_each(1) + (p - 2 * a) * one_each(0))
    return {
        "4clique": cliques,
        "tails": cliques * 4 * comb(p - 2, 2),
        # the fourth vertex of the 4-clique is the one on all three
        "on all three, one each": cliques * 4 * ((p - 2) ** 3 - (p - 2) ** 2),
        "one each": both,
    }


@pytest.mark.parametrize("p,a,b", [(6, 2, 1), (9, 3, 4), (7, 0, 3)])
def test_closed_forms_against_the_oracle(p, a, b):
    g, want = two_sides(p, a, b), totals(p, a, b)
    for name, pattern in PATTERNS.items():
        assert oracle.count(g.nindex, g.nlist, fsgc.preprocess(*pattern).to_bytes())["raw"] == want[name], name


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2048, 2049, 2300, 6000, 8192, 8193])
def test_two_sides(ctx, p):
    a, b = 4, 3
    want = totals(p, a, b)
    gid = ctx.upload(two_sides(p, a, b))
    try:
        for name, pattern in PATTERNS.items():
            mo = fsgc.preprocess(*pattern)
            assert ctx.count(gid, mo).raw_total == want[name] & M64, name
            if p in (2049, 8193):
                assert ctx.count_exact(gid, mo).raw_total == want[name], name
    finally:
        ctx.release(gid)


def clique_edges(k, first=0):
    i, j = np.triu_indices(k, 1)
    return np.stack([i, j], 1) + first


@pytest.mark.gpu
def test_clique_of_more_than_2048_out_neighbours(ctx):
    k = 2237
    gid = ctx.upload(fsgc.csr_from_edges(k, clique_edges(k)))
    try:
        assert ctx.count(gid, fsgc.preprocess(*EXTRA["4clique"])).raw_total == comb(k, 4)
        tails = comb(k, 4) * 4 * comb(k - 4, 2)
        assert ctx.count(gid, fsgc.preprocess(*EXTRA["tailed_4clique_2"])).raw_total == tails & M64
    finally:
        ctx.release(gid)


@pytest.mark.gpu
def test_supports_in_rank_order_of_packed_members(ctx):
    sizes = [1700, 40, 1650, 3]  # 2.8 M edges in all
    graphs = [fsgc.csr_from_edges(k + 5, clique_edges(k, 2)) for k in sizes]
    graphs.append(fsgc.gen_rmat(9, 8, seed=3))
    # an edge, two of its shared neighbours, one further fringe on each end
    shared = (6, [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (0, 4), (1, 5)])
    pid = ctx.upload_packed(graphs)
    try:
        for n, e in ((3, [(0, 1), (0, 2), (1, 2)]), shared):
            mo = fsgc.preprocess(n, e)
            got = ctx.count_packed(pid, mo)
            for k, r in zip(sizes, got):
                want = comb(k, 3) if n == 3 else comb(k, 2) * comb(k - 2, 2) * (k - 4) * (k - 5)
                if n > 3 and k < 6:
                    want = 0
                assert (r.count if n == 3 else r.raw_total) == want & M64, (n, k)
            g = graphs[-1]
            assert got[-1].raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"]
    finally:
        ctx.release(pid)
