"""The arena that a triangle count is admitted with is the arena it takes: none where
the bitmap rows fit in shared memory."""
import pytest

import fsgc
from helpers import EXTRA, WORKLOAD

pytestmark = pytest.mark.gpu


def clique_with_leaves(c, leaves):
    pairs = [(i, j) for i in range(c) for j in range(i + 1, c)]
    pairs += [(i, c + i * leaves + t) for i in range(c) for t in range(leaves)]
    return fsgc.csr_from_edges(c * (leaves + 1), pairs)


@pytest.mark.parametrize("c,leaves,spills", [(20, 5, False), (300, 2, False), (300, 3000, True), (700, 0, False)])
def test_triangle_footprint_is_what_a_lane_takes(ctx, c, leaves, spills):
    gid = ctx.upload(clique_with_leaves(c, leaves))
    try:
        for pattern in (EXTRA["triangle_mixed"], WORKLOAD["4clique_3_distinct"], EXTRA["4clique"]):
            mo = fsgc.preprocess(*pattern)
            need = fsgc.task_footprint(ctx, gid, mo)
            lane = fsgc.Lane(ctx)
            lane.submit([(gid, mo)])
            lane.wait()
            assert fsgc.lib().fsgc_lane_scratch_bytes(lane.ptr) == need
            assert (need > 0) == (spills and pattern is not EXTRA["4clique"])
            lane.close()
    finally:
        ctx.release(gid)
