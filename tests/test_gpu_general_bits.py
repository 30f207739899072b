"""General cores on the adjacency bit matrix of a small graph against the list
kernel: the same graph padded with isolated vertices past the matrix's limit
has the same counts.  Sizes around the matrix's word and row padding, patterns
with one to three single fringes (inclusion-exclusion) and with more (placement
walk), u64, exact and exact-placement counts."""
import numpy as np
import pytest

import fsgc
import oracle
from helpers import EXTRA, golden_cases
from test_gpu_parity import GENERAL_HUB

pytestmark = pytest.mark.gpu
LIMIT = 4096


def padded(g, n):
    return fsgc.Graph(np.concatenate([g.nindex, np.full(n - g.n, g.m)]), g.nlist)


def patterns():
    pats = [fsgc.preprocess(n, e) for n, e in {**GENERAL_HUB, "house": EXTRA["house"]}.values()]
    pats += [fsgc.MatchingOrder.from_bytes(bytes.fromhex(c["mo"])) for c in golden_cases("random")
             if c["mo"] is not None and bytes.fromhex(c["mo"])[0] >= 4][:25]
    # single fringes whose last anchor set is all anchors: the walk counts them twice
    pats += [fsgc.MatchingOrder.from_bytes(bytes.fromhex(c["mo"])) for c in golden_cases("random")
             if c["name"] in ("r130-4-path", "r300-4-path", "r375-5-cycle")]
    # two fringes on one anchor set: the reference's walk differs from the exact sum
    pats.append(fsgc.preprocess(7, [(0, 1), (1, 2), (2, 3), (3, 0), (4, 0), (4, 1), (5, 0), (5, 1), (6, 2), (6, 3)]))
    return [mo for mo in pats if mo.nodes >= 4]


@pytest.mark.parametrize("n,m", [(20, 60), (33, 110), (127, 400), (600, 1500)])
def test_bit_matrix_equals_lists(ctx, n, m):
    g = fsgc.gen_er(n, m, seed=n)
    a, b = ctx.upload(g), ctx.upload(padded(g, LIMIT + 1))
    try:
        pats = patterns()
        assert len(pats) >= 20
        for exact in (False, True):
            ctx.set_exact_placements(exact)
            for i, mo in enumerate(pats):
                x, y = ctx.count(a, mo), ctx.count(b, mo)
                if x.flags:  # the pattern is larger than the small graph
                    continue
                assert (x.raw_total, x.automorphisms, x.core_type) == (y.raw_total, y.automorphisms, y.core_type), (i, exact)
        for mo in pats[:8]:
            if not ctx.count(a, mo).flags:
                assert ctx.count_exact(a, mo).raw_total == ctx.count_exact(b, mo).raw_total
    finally:
        ctx.set_exact_placements(False)
        ctx.release(a)
        ctx.release(b)


def test_largest_bit_matrix(ctx):
    g = padded(fsgc.gen_er(700, 2100, 9), LIMIT)
    gid = ctx.upload(g)
    try:
        for name in ("5cycle", "5cycle_chord_fringe", "4path_ends"):
            mo = fsgc.preprocess(*GENERAL_HUB[name])
            assert ctx.count(gid, mo).raw_total == oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"], name
    finally:
        ctx.release(gid)
