"""Pattern sets with edge patterns that no edge of the graph has degrees for: left out,
and counted as nothing, on both sides of the limits."""
import numpy as np
import pytest

import fsgc
import oracle

pytestmark = pytest.mark.gpu


def pattern(f_u, f_v, f_uv):
    e, n = [(0, 1)], 2
    for ends, f in (((0,), f_u), ((1,), f_v), ((0, 1), f_uv)):
        for _ in range(f):
            e += [(a, n) for a in ends]
            n += 1
    return fsgc.preprocess(n, e)


def regular(n, d):
    """Every vertex joined to the d / 2 before and after it."""
    i = np.arange(n)
    return fsgc.csr_from_edges(n, np.concatenate([np.stack([i, (i + k) % n], 1) for k in range(1, d // 2 + 1)]))


GRAPHS = [regular(50, 2), regular(50, 4), regular(60, 8),
          fsgc.csr_from_edges(40, [(0, i) for i in range(1, 40)]),
          fsgc.csr_from_edges(30, [(0, 1)] + [(0, i) for i in range(2, 9)] + [(1, i) for i in range(9, 15)])]


@pytest.mark.parametrize("i", range(len(GRAPHS)))
def test_sets_equal_the_oracle(ctx, i):
    g = GRAPHS[i]
    mos = [pattern(a, b, s) for a in range(0, 8) for b in range(max(a, 1), 8) for s in range(0, 3)]
    mos = [mo for mo in mos if mo.nodes == 2]
    want = [oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"] for mo in mos]
    assert 0 in want
    gid = ctx.upload(g)
    try:
        for call in range(3):
            assert [r.raw_total for r in ctx.count_set(gid, mos)] == want
        nothing = [mo for mo, w in zip(mos, want) if w == 0][:2]
        for call in range(3):  # a set of such patterns alone
            assert [r.raw_total for r in ctx.count_set(gid, nothing)] == [0] * len(nothing)
    finally:
        ctx.release(gid)
