"""Edge-core formulas from chains of binomials: every pair of fringe counts that
has a kernel and the first beyond, on graphs with degrees around the counts,
around the point where a subtraction replaces a division no longer, and where
the reference's binomials wrap."""
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


def hub_graph():
    """Hubs of degree 100,000 and 9,000-16,000 (C(n, 4) n and C(n, 5) n wrap there) over a sparse graph."""
    n = 100_200
    rng = np.random.default_rng(3)
    pairs = [np.stack([np.zeros(100_000, np.int64), np.arange(1, 100_001)], 1)]
    for h, d in ((100_100, 9_000), (50, 11_600), (100_150, 11_900), (7, 16_000)):
        pairs.append(np.stack([np.full(d, h), rng.choice(100_000, d, replace=False) + 1], 1))
    pairs.append(rng.integers(0, n, (60_000, 2)))
    pairs.append(np.array([(a, b) for a in (0, 7, 50, 100_100, 100_150) for b in (7, 50, 100_100, 100_150) if a != b]))
    return fsgc.csr_from_edges(n, np.concatenate(pairs))


@pytest.fixture(scope="module")
def graphs():
    return [fsgc.gen_er(60, 300, 1), fsgc.gen_er(3000, 18_000, 2), hub_graph()]


@pytest.mark.parametrize("f_u", range(8))
def test_edge_formula_chains(ctx, graphs, f_u):
    for g in graphs:
        gid = ctx.upload(g)
        try:
            for f_v in range(max(f_u, 1), 8):
                for f_uv in (0, 2):
                    mo = pattern(f_u, f_v, f_uv)
                    if mo.nodes != 2:
                        continue
                    want = oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"]
                    assert ctx.count(gid, mo).raw_total == want, (g.n, f_u, f_v, f_uv)
                    assert ctx.count_set(gid, [mo, mo])[0].raw_total == want, (g.n, f_u, f_v, f_uv)
        finally:
            ctx.release(gid)
