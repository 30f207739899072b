"""A graph whose rank-ordered copy finds no room is counted without it, is not asked
for it again while no more room is there, and has it once there is."""
import pytest

import fsgc

pytestmark = pytest.mark.gpu
WEDGES = [(5, [(0, 1), (0, 2), (1, 3), (2, 4)]), (7, [(0, 1), (0, 2), (1, 3), (1, 4), (2, 5), (2, 6)])]


def test_the_copy_is_tried_again_when_there_is_room(ctx):
    torch = pytest.importorskip("torch")
    mos = [fsgc.preprocess(*w) for w in WEDGES]
    g = fsgc.gen_er(1_000_000, 8_000_000, 5)
    gid = ctx.upload(g)
    copy = 10 * g.m  # bytes; twice that more while it is built
    filler = None
    try:
        ctx.prepare(gid)
        ctx.lean(gid)
        want = [r.raw_total for r in ctx.count_batch([(gid, mo) for mo in mos])]
        before = ctx.info(gid).device_bytes
        ctx.lean(gid, False)
        free, _ = torch.cuda.mem_get_info()
        filler = torch.empty(free - (2 * copy - (32 << 20)), dtype=torch.uint8, device="cuda")
        steps = []
        for call in range(4):
            at = ctx.launches
            assert [r.raw_total for r in ctx.count_set(gid, mos)] == want, call
            steps.append(ctx.launches - at)
            assert ctx.info(gid).device_bytes == before and fsgc.lib().fsgc_graph_fast_bytes(ctx.ptr, gid) == 0
        assert steps[3] == 1  # a captured set, replayed
        assert [ctx.count(gid, mo).raw_total for mo in mos] == want
        del filler
        filler = None
        torch.cuda.empty_cache()
        for call in range(4):
            assert [r.raw_total for r in ctx.count_set(gid, mos)] == want, call
            assert ctx.info(gid).device_bytes >= before + copy
        assert [ctx.count(gid, mo).raw_total for mo in mos] == want
    finally:
        del filler
        torch.cuda.empty_cache()
        ctx.release(gid)
