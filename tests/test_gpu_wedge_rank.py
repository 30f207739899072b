"""The rank-order wedge path against the oracle: every way a rank-order owner is
counted (one warp's table, the block's table, counters of 2 to 32 bits, owners
with more centres than one batch), residuals of every kind (none, 4-cycles,
mixed, two and more fringes, wrapping binomials whose value depends on which
end has the larger id), single, fused, packed and exact counts.  Counts are
whole numbers: equality, no tolerance."""
import numpy as np
import pytest

import fsgc
import oracle

pytestmark = pytest.mark.gpu

W = [(0, 1), (0, 2)]


def ends(a, b, shared=0):
    """Wedge with a and b fringes on its ends and `shared` on both."""
    e, v = list(W), 3
    for at, k in ((1, a), (2, b)):
        for _ in range(k):
            e.append((at, v))
            v += 1
    for _ in range(shared):
        e += [(1, v), (2, v)]
        v += 1
    return v, e


def order(a, b, shared=0):
    """The matching order with these fringe counts (A is the centre), as a
    caller may pass it; the decomposition gives the same core for most."""
    mo = fsgc.MatchingOrder()
    mo.nodes = 3
    mo.list[0], mo.list[1] = 1, 1
    sets = [(2, a), (4, b), (6, shared)]
    for at, k in sets:
        if k:
            mo.anch[mo.anchorsets], mo.fcnt[mo.anchorsets] = at, k
            mo.anchorsets += 1
    return mo


KINDS = [(1, 1, 0), (0, 0, 1), (1, 1, 1), (3, 1, 0), (2, 2, 0), (0, 0, 2), (1, 0, 1), (4, 4, 0), (7, 7, 0), (2, 1, 2)]


def sparse_hubs():
    """Ids far apart: hubs of degree 2,600, 900 and 300 over 300,000 ids, so
    that owners sweep several chunks and read the boundary table."""
    rng = np.random.default_rng(5)
    n = 300000
    pairs = [(h, int(x)) for h, k in ((7, 2600), (150000, 900), (299999, 300)) for x in rng.choice(n, k, replace=False)
             if x != h]
    pairs += list(zip(rng.integers(0, n, 60000).tolist(), rng.integers(0, n, 60000).tolist()))
    return fsgc.csr_from_edges(n, pairs)


def twin_hubs(leaves, path):
    """Two hubs that share `leaves` neighbours (32-bit counters from 65,536),
    and a path over the first of them."""
    pairs = [(h, i) for h in (0, 1) for i in range(2, leaves + 2)] + [(i, i + 1) for i in range(2, path)]
    return fsgc.csr_from_edges(leaves + 70, pairs)


GRAPHS = {
    "er": lambda: fsgc.gen_er(4000, 24000, 3),
    "er_dense": lambda: fsgc.gen_er(220, 11000, 4),
    "rmat": lambda: fsgc.gen_rmat(10, 16, seed=6),
    "cl": lambda: fsgc.gen_chung_lu(4000, 12.0, 2.3, 8),
    "sparse_hubs": sparse_hubs,
}


@pytest.mark.parametrize("gname", list(GRAPHS))
def test_rank_order_counts_match_oracle(ctx, gname):
    g = GRAPHS[gname]()
    assert g.m >= 20000
    gid = ctx.upload(g)
    try:
        mos = [order(*k) for k in KINDS]
        want = []
        for k, mo in zip(KINDS, mos):
            o = oracle.count(g.nindex, g.nlist, mo.to_bytes())
            r = ctx.count(gid, mo)
            assert (r.raw_total, r.count, r.automorphisms, r.core_type) == (o["raw"], o["count"], o["aut"], o["core"]), k
            want.append(r)
        for call in range(3):  # fused passes: direct, captured, replayed
            for k, a, b in zip(KINDS, ctx.count_set(gid, mos), want):
                assert (a.raw_total, a.count) == (b.raw_total, b.count), (call, k)
        for k, mo in list(zip(KINDS, mos))[:6]:
            x, o = ctx.count_exact(gid, mo), oracle.count_exact(g.nindex, g.nlist, mo.to_bytes())
            assert (x.raw_total, x.saturated) == (o["raw"], o["saturated"]), k
    finally:
        ctx.release(gid)


def test_rank_order_wide_counters(ctx):
    """Hub owners with more centres than a batch, and counts too large for a
    staged pair (16,384) or for 16 bits (closed forms on K(2, 66000))."""
    g = twin_hubs(17000, 60)
    gid = ctx.upload(g)
    try:
        for k in [(0, 0, 1), (1, 1, 1), (0, 0, 2), (3, 1, 0), (2, 2, 1)]:
            mo = order(*k)
            o = oracle.count(g.nindex, g.nlist, mo.to_bytes())
            assert ctx.count(gid, mo).raw_total == o["raw"], k
    finally:
        ctx.release(gid)
    L = 66000
    gid = ctx.upload(twin_hubs(L, 0))
    try:
        # pairs: the hubs share L neighbours, every two leaves share 2
        hub, leaf = L, L * (L - 1) // 2
        assert ctx.count(gid, order(0, 0, 1)).raw_total == hub * (L - 1) + leaf * 2
        assert ctx.count(gid, order(0, 0, 2)).raw_total == hub * (L - 1) * (L - 2) // 2
        # one fringe on each end: C ((dx - 1) (dy - 1) - (C - 1))
        assert ctx.count(gid, order(1, 1, 0)).raw_total == hub * ((L - 1) ** 2 - (L - 1))
    finally:
        ctx.release(gid)


def test_rank_order_packed_members(ctx):
    graphs = [fsgc.gen_er(3000, 9000, 1), fsgc.gen_rmat(9, 8, seed=2), fsgc.csr_from_edges(1, []),
              fsgc.gen_chung_lu(2500, 8.0, 2.2, 4), fsgc.csr_from_edges(3000, [(2999, i) for i in range(2600)])]
    pid = ctx.upload_packed(graphs)
    try:
        for k in KINDS:
            mo = order(*k)
            for g, r in zip(graphs, ctx.count_packed(pid, mo)):
                o = oracle.count(g.nindex, g.nlist, mo.to_bytes())
                assert (r.raw_total, r.count) == (o["raw"], o["count"]), (k, g.n)
    finally:
        ctx.release(pid)
