"""What a served graph must hold, and what is given up where the budget is short:
no chunk table beside a copy in rank order, and registration and admission within
the bytes of the derived structures alone.  Counts are the same either way."""
import ctypes as C

import pytest

import fsgc
import oracle
from helpers import EXTRA, WORKLOAD

pytestmark = pytest.mark.gpu
WEDGE = WORKLOAD["wedge_1_on_each_end"]
CYCLE = WORKLOAD["4cycle_opposite"]


def base_bytes(g):
    """Graph, orientation, supports, per-vertex triangles and per-entry supports."""
    return 8 * (g.n + 1) + 4 * (g.m + g.n) + 8 * (g.n + 1) + 3 * 4 * (g.m // 2) + 8 * g.n + 4 * g.m


def test_no_chunk_table_beside_the_copy_in_rank_order(ctx):
    g = fsgc.gen_er(40_000, 160_000, 3)  # no list is long enough for a table row or a wide block
    gid = ctx.upload(g)
    try:
        ctx.prepare_all(gid)
        copy = 4 * (3 * g.n + 2 + 2 * g.m) + 2 * g.m
        slack = 65536  # boundary rows of the few long lists; a chunk table has 8 bytes a vertex
        assert ctx.info(gid).device_bytes <= base_bytes(g) + copy + slack < base_bytes(g) + copy + 8 * g.n
        fast = fsgc.lib().fsgc_graph_fast_bytes(ctx.ptr, gid)
        assert fast >= copy
        ctx.lean(gid)
        assert fsgc.lib().fsgc_graph_fast_bytes(ctx.ptr, gid) == 0
        assert ctx.info(gid).device_bytes <= base_bytes(g)
    finally:
        ctx.release(gid)


@pytest.mark.parametrize("g", [fsgc.gen_er(40_000, 160_000, 3), fsgc.gen_er(3000, 12_000, 9),
                               fsgc.gen_chung_lu(20_000, 8.0, 2.3, 5)], ids=["er", "small", "hubs"])
def test_lean_counts_are_equal(ctx, g):
    """Single counts, sets (direct, captured, replayed) and lanes, before, while and
    after a graph goes without the faster structures."""
    pats = {"wedge": WEDGE, "4cycle": CYCLE, "two": (7, [(0, 1), (0, 2), (1, 3), (1, 4), (2, 5), (2, 6)]),
            "triangle": EXTRA["triangle_mixed"]}
    if g.n <= 4096:
        pats["centre"] = EXTRA["wedge_centre_and_ends"]
        pats["general"] = EXTRA["5cycle"]
    mos = [fsgc.preprocess(*p) for p in pats.values()]
    want = [oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"] for mo in mos]
    gid = ctx.upload(g)
    lane = fsgc.Lane(ctx)
    try:
        for on in (False, True, False):
            ctx.lean(gid, on)
            assert [ctx.count(gid, mo).raw_total for mo in mos] == want
            for call in range(3):
                assert [r.raw_total for r in ctx.count_set(gid, mos)] == want, (on, call)
            lane.submit([(gid, mo) for mo in mos])
            assert [r.raw_total for r in lane.wait()] == want
            assert ctx.count_exact(gid, mos[0]).raw_total % (1 << 64) == want[0]
            assert (fsgc.lib().fsgc_graph_fast_bytes(ctx.ptr, gid) > 0) != on
    finally:
        lane.close()
        ctx.release(gid)


def test_registration_and_admission_without_the_faster_structures(ctx):
    graphs = [fsgc.gen_er(40_000, 160_000, seed) for seed in (3, 4)]
    gids = [ctx.upload(g) for g in graphs]
    mo = fsgc.preprocess(*WEDGE)
    want = [oracle.count(g.nindex, g.nlist, mo.to_bytes())["raw"] for g in graphs]
    lean, full = [], []
    try:
        for gid in gids:
            ctx.lean(gid)
            ctx.prepare_all(gid)
            lean.append(ctx.info(gid).device_bytes)
            ctx.lean(gid, False)
            ctx.prepare_all(gid)
            full.append(ctx.info(gid).device_bytes)
            assert full[-1] > lean[-1] + 3_000_000

        def served(srv):
            return [srv.wait(srv.submit(gid, mo), timeout_s=60)[0].raw_total for gid in gids]

        with fsgc.Server(ctx, memory_budget=sum(lean), lanes=2, max_batch=4) as srv:
            for gid in gids:
                srv.add_graph(gid)
            srv.add_graph(gids[0])  # again: nothing changes
            assert srv.stats().in_use_bytes <= sum(lean)
            assert served(srv) == want
            assert [ctx.info(gid).device_bytes for gid in gids] == lean
        # the graphs may be fast again once the server is gone
        assert [ctx.count(gid, mo).raw_total for gid in gids] == want
        assert all(fsgc.lib().fsgc_graph_fast_bytes(ctx.ptr, gid) > 0 for gid in gids)
        # the first registered gives way to the second, but not to what cannot fit
        with fsgc.Server(ctx, memory_budget=full[0] + lean[1], lanes=1, max_batch=4) as srv:
            for gid in gids:
                srv.add_graph(gid)
            assert srv.stats().in_use_bytes <= full[0] + lean[1]
            assert served(srv) == want
        with fsgc.Server(ctx, memory_budget=full[0] + lean[1] - 1, lanes=1, max_batch=4) as srv:
            srv.add_graph(gids[0])
            srv.add_graph(gids[1])
            assert srv.stats().in_use_bytes == sum(lean)
        with fsgc.Server(ctx, memory_budget=sum(lean) - 1, lanes=1, max_batch=4) as srv:
            srv.add_graph(gids[0])
            with pytest.raises(fsgc.FsgcError):
                srv.add_graph(gids[1])
    finally:
        for gid in gids:
            ctx.release(gid)


def test_a_query_that_fits_only_beside_lean_graphs(ctx):
    """A hub graph: its wedge count needs an arena."""
    hub = fsgc.csr_from_edges(30_000, [(0, i) for i in range(1, 15_000)] + [(1, i) for i in range(2, 15_000)])
    mo = fsgc.preprocess(*WEDGE)
    want = oracle.count(hub.nindex, hub.nlist, mo.to_bytes())["raw"]
    gid = ctx.upload(hub)
    try:
        need = fsgc.task_footprint(ctx, gid, mo)
        ctx.lean(gid)
        ctx.prepare_all(gid)
        lean = ctx.info(gid).device_bytes
        ctx.lean(gid, False)
        ctx.prepare_all(gid)
        full = ctx.info(gid).device_bytes
        assert need > 0 and full > lean
        with fsgc.Server(ctx, memory_budget=lean + need, lanes=2, max_batch=1) as srv:
            srv.add_graph(gid)
            assert ctx.info(gid).device_bytes == full  # fits by itself
            assert srv.wait(srv.submit(gid, mo), timeout_s=60)[0].raw_total == want
            assert srv.stats().in_use_bytes <= lean + need
            assert ctx.info(gid).device_bytes == lean
        with fsgc.Server(ctx, memory_budget=lean + need - 1, lanes=2, max_batch=1) as srv:
            srv.add_graph(gid)
            t = C.c_uint64()
            assert fsgc.lib().fsgc_server_submit(srv.ptr, gid, C.byref(mo), C.byref(t)) == 8  # FSGC_EBUSY
            assert ctx.info(gid).device_bytes == full  # and nothing was given up for it
    finally:
        ctx.release(gid)
