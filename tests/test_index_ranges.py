"""Sizes up to which 32-bit indices are used: a grid-stride step past the last item
must not pass 2^31 - 1 (an overflowed index is negative and read through)."""
import ctypes as C

import fsgc

STEP = 16 * 1024 * 256  # blocks an SM, SMs, threads: no GPU launches more of these kernels
INT_MAX = 2**31 - 1


def ordered(edges, n, squares_per_edge):
    f = fsgc.lib().fsgc_supports_ordered_host
    f.argtypes = [C.c_longlong, C.c_int, C.c_ulonglong]
    return bool(f(edges, n, edges * squares_per_edge))


def test_ordered_supports_keep_their_indices_in_range():
    assert ordered(3_000_000, 100_000, 50) and not ordered(3_000_000, 100_000, 30)
    assert not ordered(2_000_000, 100_000, 50)
    lo, hi = 3_000_000, 2**32  # the largest number of edges that is taken
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if ordered(mid, 100_000, 50) else (lo, mid)
    assert lo > 2**30 and lo + STEP <= INT_MAX
    lo, hi = 100_000, 2**31 - 1
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if ordered(3_000_000, mid, 50) else (lo, mid)
    assert lo > 2**30 and lo + STEP <= INT_MAX
