"""Wedges with a fringed centre on the adjacency bit matrix of a small graph
against the list kernel: the same graph padded with isolated vertices past the
matrix's limit has the same counts.  Sizes around a lane's one, two and four
words of a row, fringes on every anchor set, closed and open wedges, and a hub
whose binomials wrap."""
import numpy as np
import pytest

import fsgc
import oracle

pytestmark = pytest.mark.gpu
LIMIT = 4096
CENTRE, ENDS = 0, (1, 2)
SETS = [(0,), (1,), (2,), (0, 1), (0, 2), (1, 2), (0, 1, 2)]
FRINGES = [(1, 0, 0, 0, 0, 0, 0), (1, 1, 1, 0, 0, 0, 0), (2, 1, 0, 0, 0, 0, 0), (1, 0, 3, 1, 0, 0, 0),
           (0, 0, 1, 2, 1, 0, 0), (2, 2, 2, 0, 0, 2, 0), (0, 1, 0, 0, 0, 1, 1), (1, 2, 1, 1, 2, 1, 1), (1, 1, 1, 0, 0, 0, 2), (1, 0, 1, 0, 0, 0, 0), (7, 1, 1, 0, 0, 0, 0)]


def patterns():
    pats = []
    for fr in FRINGES:
        e, n = [(0, 1), (0, 2)], 3
        for ends, f in zip(SETS, fr):
            for _ in range(f):
                e += [(a, n) for a in ends]
                n += 1
        mo = fsgc.preprocess(n, e)
        if mo.nodes == 3:
            pats.append(mo)
    assert len(pats) >= 5
    return pats


def padded(g, n):
    return fsgc.Graph(np.concatenate([g.nindex, np.full(n - g.n, g.m)]), g.nlist)


def hub(n):
    pairs = [(0, i) for i in range(1, n)]
    pairs += np.random.default_rng(n).integers(0, n, (3 * n, 2)).tolist()
    return fsgc.csr_from_edges(n, pairs)


@pytest.mark.parametrize("g", [fsgc.gen_er(40, 200, 1), fsgc.gen_er(1024, 6000, 2), fsgc.gen_er(1025, 6000, 3),
                               fsgc.gen_er(2048, 9000, 4), fsgc.gen_er(2049, 9000, 5), hub(700),
                               padded(fsgc.gen_er(900, 9000, 6), LIMIT)], ids=lambda g: f"n{g.n}")
def test_wedge_bits_equal_lists(ctx, g):
    a, b = ctx.upload(g), ctx.upload(padded(g, LIMIT + 1))
    try:
        for i, mo in enumerate(patterns()):
            x, y = ctx.count(a, mo), ctx.count(b, mo)
            assert (x.raw_total, x.automorphisms) == (y.raw_total, y.automorphisms), i
            if i < 3:
                assert x.raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"], i
                assert ctx.count_exact(a, mo).raw_total == ctx.count_exact(b, mo).raw_total, i
    finally:
        ctx.release(a)
        ctx.release(b)
