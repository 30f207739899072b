"""Wedges with all fringes on one end, counted in rank order on graphs whose
hubs make the binomials wrap: the pair formula then depends on the number of
centres, which it does not while nothing wraps.  Whole numbers: equality with the
oracle, for single counts and sets."""
import numpy as np
import pytest

import fsgc
import oracle

pytestmark = pytest.mark.gpu


def order(a, b):
    """Matching order of a wedge with a and b fringes on its ends (the centre
    first), as a caller may pass it."""
    mo = fsgc.MatchingOrder()
    mo.nodes = 3
    mo.list[0], mo.list[1] = 1, 1
    for at, k in ((2, a), (4, b)):
        if k:
            mo.anch[mo.anchorsets], mo.fcnt[mo.anchorsets] = at, k
            mo.anchorsets += 1
    return mo


def hubs(degrees):
    """Hubs over 60,000 ids whose neighbourhoods overlap, and a sparse rest."""
    rng = np.random.default_rng(11)
    n = 60000
    pairs = [np.stack([np.full(k, 7 + 20000 * i), rng.choice(6000, k, replace=False) + 30000], 1)
             for i, k in enumerate(degrees)]
    pairs.append(rng.integers(0, n, (20000, 2)))
    return fsgc.csr_from_edges(n, np.concatenate(pairs))


@pytest.mark.parametrize("degrees", [(2600, 900, 300), (4200, 2600, 40), (700, 90, 30)])
def test_one_sided_fringes(ctx, degrees):
    g = hubs(degrees)
    assert g.m >= 20000
    gid = ctx.upload(g)
    try:
        kinds = [(1, 0), (3, 0), (0, 5), (7, 0), (0, 7), (9, 0), (12, 0)]
        mos = [order(*k) for k in kinds]
        want = [oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"] for mo in mos]
        assert [ctx.count(gid, mo).raw_total for mo in mos] == want
        for call in range(3):  # direct, captured, replayed
            assert [r.raw_total for r in ctx.count_set(gid, mos)] == want, call
    finally:
        ctx.release(gid)
