"""The rank-ordered copy of graphs with long lists, which the whole grid passes over:
hubs on both sides of the line, more hubs than one, hubs of packed members; first
counts, which build the copy, against the oracle or closed forms."""
import numpy as np
import pytest

import fsgc
import oracle

pytestmark = pytest.mark.gpu
ENDS = (5, [(0, 1), (0, 2), (1, 3), (2, 4)])
TWO = (7, [(0, 1), (0, 2), (1, 3), (1, 4), (2, 5), (2, 6)])


def hubs(n, degrees, rest, seed=7):
    rng = np.random.default_rng(seed)
    pairs = [np.stack([np.full(k, n - 1 - 3 * i), rng.choice(n - 40, k, replace=False)], 1) for i, k in enumerate(degrees)]
    return fsgc.csr_from_edges(n, np.concatenate(pairs + [rng.integers(0, n, (rest, 2))]))


@pytest.mark.parametrize("degrees", [(4096,), (4097,), (12000,), (4500, 4216, 4215, 4100), (9000, 8000, 5000, 1000, 40)])
def test_hubs(ctx, degrees):
    g = hubs(15_000, degrees, 9000)
    gid = ctx.upload(g)
    try:
        for p in (ENDS, TWO):
            mo = fsgc.preprocess(*p)
            assert ctx.count(gid, mo).raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"]
    finally:
        ctx.release(gid)


@pytest.mark.parametrize("leaves", [30_000, 700_000])
def test_one_hub_over_a_path(ctx, leaves):
    """A hub joined to every vertex of a path: its list and the linear sums over it
    in closed form."""
    L = leaves
    g = fsgc.csr_from_edges(L + 1, np.concatenate([np.stack([np.full(L, L), np.arange(L)], 1),
                                                   np.stack([np.arange(L - 1), np.arange(1, L)], 1)]))
    gid = ctx.upload(g)
    try:
        # 4-cycles: every path of three vertices closes over the hub
        c4 = fsgc.preprocess(4, [(0, 1), (1, 2), (2, 3), (3, 0)])
        assert ctx.count(gid, c4).count == L - 2
        # paths of three edges, counted as wedges with a fringe on one end: over the
        # middle edge, less three times the triangles
        d = g.degrees().astype(object)
        mo = fsgc.MatchingOrder()
        mo.nodes, mo.anchorsets = 3, 1
        mo.list[0], mo.list[1], mo.anch[0], mo.fcnt[0] = 1, 1, 2, 1
        src = np.repeat(np.arange(g.n), g.degrees())
        once = src < g.nlist
        want = int(sum((d[src[once]] - 1) * (d[g.nlist[once]] - 1))) - 3 * (L - 1)
        assert ctx.count(gid, mo).count == want
    finally:
        ctx.release(gid)


def test_hubs_of_packed_members(ctx):
    graphs = [hubs(9000, (5000,), 3000), fsgc.gen_er(2000, 6000, 1), hubs(12_000, (7000, 4300), 3000)]
    pid = ctx.upload_packed(graphs)
    try:
        for p in (ENDS, TWO):
            mo = fsgc.preprocess(*p)
            got = [r.raw_total for r in ctx.count_packed(pid, mo)]
            assert got == [oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"] for g in graphs]
    finally:
        ctx.release(pid)
