"""Exact wedge counts whose pairs are evaluated one by one, on dense graphs (counted by
chunks) and beside them (in rank order), and where the u64 count wraps."""
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


GRAPHS = {"dense": lambda: fsgc.gen_er(500, 14_000, 1), "clique": lambda: clique(160), "sparse": lambda: fsgc.gen_er(4000, 12_000, 4),
          "rmat": lambda: fsgc.gen_rmat(10, 16, seed=3)}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_exact_counts(ctx, name):
    g = GRAPHS[name]()
    gid = ctx.upload(g)
    try:
        for k in [(2, 2, 0), (5, 4, 0), (8, 7, 0), (9, 9, 3), (3, 1, 0), (9, 0, 0), (2, 1, 1)]:
            mo = order(*k)
            x, o = ctx.count_exact(gid, mo), oracle.count_exact(g.nindex, g.nlist, mo.to_bytes())
            assert x.saturated == o["saturated"], k
            if not x.saturated:  # the oracle gives no total then
                assert x.raw_total == o["raw"], k
    finally:
        ctx.release(gid)
