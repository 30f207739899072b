"""Vertex counts that 32-bit vertex loops cannot walk are refused before anything is
allocated or launched."""
import ctypes as C

import numpy as np
import pytest

import fsgc

pytestmark = pytest.mark.gpu
LIMIT = 2**31 - 1 - 2**22


@pytest.mark.parametrize("n", [LIMIT + 1, 2**31 - 1])
def test_graphs_of_too_many_vertices_are_refused(ctx, n):
    with pytest.raises(fsgc.FsgcError):
        ctx.upload_edges(n, np.zeros((0, 2), np.int32))
    assert b"vertices" in fsgc.lib().fsgc_ctx_last_error(ctx.ptr)
    # refused before the arrays are looked at
    off, gid = (C.c_int64 * 2)(0, 0), C.c_int()
    for name in ("fsgc_graph_from_csr", "fsgc_graph_from_device_csr"):
        assert getattr(fsgc.lib(), name)(ctx.ptr, n, C.c_int64(0), off, None, C.byref(gid)) == 5, name
    off32 = (C.c_int32 * 2)(0, 0)
    assert fsgc.lib().fsgc_graph_from_csr32(ctx.ptr, n, 0, off32, None, C.byref(gid)) == 5
    # the context goes on
    g = fsgc.csr_from_edges(4, [(0, 1), (1, 2), (0, 2), (2, 3)])
    small = ctx.upload(g)
    assert ctx.count(small, fsgc.preprocess(3, [(0, 1), (1, 2), (0, 2)])).count == 1
    ctx.release(small)
