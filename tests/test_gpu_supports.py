"""Edge supports on both sides of the rule by which lists are put in rank order:
out-degrees above a warp's table and above a block's (cliques, in closed form),
in-edges of several pieces (hubs), isolated ends, against the oracle's edge
counts."""
from math import comb

import numpy as np
import pytest

import fsgc
import oracle

pytestmark = pytest.mark.gpu
SHARED = (6, [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (0, 4), (1, 5)])  # two fringes on both, one on each


def clique(k, n):
    a, b = np.triu_indices(k, 1)
    return fsgc.csr_from_edges(n, np.stack([a, b], 1) + (n - k) // 2)


@pytest.mark.parametrize("k", [2236, 2237, 2600])
def test_cliques(ctx, k):
    gid = ctx.upload(clique(k, k + 50))
    try:
        assert ctx.count(gid, fsgc.preprocess(3, [(0, 1), (0, 2), (1, 2)])).count == comb(k, 3)
        # an edge, two of the k - 2 shared neighbours, one further fringe on each end
        want = comb(k, 2) * comb(k - 2, 2) * (k - 4) * (k - 5)
        assert want > 1 << 64  # the counts are modulo 2^64
        assert ctx.count(gid, fsgc.preprocess(*SHARED)).raw_total == want % (1 << 64)
    finally:
        ctx.release(gid)


def hubs(n):
    rng = np.random.default_rng(n)
    pairs = [np.stack([np.full(n - 10, h), np.arange(n - 10)], 1) for h in (3, n // 2, n - 11)]
    pairs.append(rng.integers(0, n - 10, (3 * n, 2)))
    pairs.append(np.stack([rng.integers(0, n // 20, 60 * n), rng.integers(0, n // 4, 60 * n)], 1))
    return fsgc.csr_from_edges(n, np.concatenate(pairs))


@pytest.mark.parametrize("g", [fsgc.gen_er(300_000, 2_600_000, 1), hubs(60_000)],
                         ids=["short lists", "hubs"])
def test_supports_against_oracle(ctx, g):
    gid = ctx.upload(g)
    try:
        for n, e in ((3, [(0, 1), (0, 2), (1, 2)]), SHARED):
            mo = fsgc.preprocess(n, e)
            assert ctx.count(gid, mo).raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"]
    finally:
        ctx.release(gid)
