"""Wedges whose pairs are evaluated one by one, on graphs on both sides of the rule by
which they are counted by chunks instead of in rank order, alone and in sets with
patterns that stay in rank order: single, batched, captured, replayed, on lanes of a
fresh graph, packed, exact, and without the copy.  Whole numbers: equality with the
oracle."""
import numpy as np
import pytest

import fsgc
import oracle

pytestmark = pytest.mark.gpu


def order(a, b, shared=0):
    mo = fsgc.MatchingOrder()
    mo.nodes = 3
    mo.list[0], mo.list[1] = 1, 1
    for at, k in ((2, a), (4, b), (6, shared)):
        if k:
            mo.anch[mo.anchorsets], mo.fcnt[mo.anchorsets] = at, k
            mo.anchorsets += 1
    return mo


def clique(k):
    i, j = np.triu_indices(k, 1)
    return fsgc.csr_from_edges(k, np.stack([i, j], 1))


GRAPHS = {
    "dense": lambda: fsgc.gen_er(600, 15_000, 1),
    "sets only": lambda: fsgc.gen_er(1500, 12_000, 2),
    "clique": lambda: clique(150),
    "clique, large": lambda: clique(280),
    "rmat": lambda: fsgc.gen_rmat(10, 16, seed=3),
    "sparse": lambda: fsgc.gen_er(4000, 12_000, 4),
}
KINDS = [(2, 2, 0), (3, 3, 0), (3, 2, 1), (3, 1, 0), (1, 1, 0), (0, 0, 2), (2, 1, 1), (2, 0, 0)]


@pytest.mark.parametrize("name", list(GRAPHS))
def test_every_way_of_counting(ctx, name):
    g = GRAPHS[name]()
    assert g.m >= 20_000
    mos = [order(*k) for k in KINDS]
    want = [oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"] for mo in mos]
    lane = fsgc.Lane(ctx)
    gid = ctx.upload(g)
    try:
        lane.submit([(gid, mo) for mo in mos])
        assert [r.raw_total for r in lane.wait()] == want
        ctx.prepare_all(gid)
        for on in (False, True, False):
            ctx.lean(gid, on)
            assert [ctx.count(gid, mo).raw_total for mo in mos] == want
            assert [r.raw_total for r in ctx.count_batch([(gid, mo) for mo in mos])] == want
            for size in (1, 2, 3, len(mos)):
                for call in range(3):
                    assert [r.raw_total for r in ctx.count_set(gid, mos[:size])] == want[:size], (on, size, call)
        for mo in mos[:3]:
            x, o = ctx.count_exact(gid, mo), oracle.count_exact(g.nindex, g.nlist, mo.to_bytes())
            assert (x.raw_total, x.saturated) == (o["raw"], o["saturated"])
    finally:
        lane.close()
        ctx.release(gid)
    pid = ctx.upload_packed([g, clique(40), g])
    try:
        for mo, w in zip(mos, want):
            r = ctx.count_packed(pid, mo)
            assert [r[0].raw_total, r[2].raw_total] == [w, w]
    finally:
        ctx.release(pid)
