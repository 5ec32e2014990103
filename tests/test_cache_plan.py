"""The length tables of a growing compressed cache (nsa_cache_plan: host arithmetic, no GPU)."""
import ctypes

import pytest

from nsa_b200 import _lib


def _plan(new, old=None, block=32, stride=16, old_block=32, old_stride=16):
    """(return code, the parts of the table, info) of a cache that grows from the lengths `old` to `new`."""
    n = len(new)
    cum = lambda ls: [sum(ls[:i]) for i in range(len(ls) + 1)]
    i32 = lambda xs: (ctypes.c_int32 * len(xs))(*xs)
    table, info = (ctypes.c_int32 * (6 * n + 4))(), (ctypes.c_int32 * 3)()
    tc = lambda L: (L - old_block) // old_stride + 1 if L >= old_block else 0
    rc = _lib.lib().nsa_cache_plan(i32(cum(new)), i32(cum(old)) if old else None, i32(cum([tc(L) for L in old])) if old else None,
                                   n, block, stride, table, info)
    t = list(table)
    return rc, [t[i * (n + 1):(i + 1) * (n + 1)] for i in range(4)] + [t[4 * n + 4:5 * n + 4], t[5 * n + 4:]], list(info)


def test_plan_of_a_growing_cache():
    rc, (cu, cc, old, row, first, order), info = _plan([40, 20, 64, 5], [31, 20, 48, 0])
    assert rc == 0 and cu == [0, 40, 60, 124, 129] and cc == [0, 1, 1, 4, 4] and old == [0, 0, 0, 2, 2]
    assert row == [0, 1, 1, 2, 2] and first == [0, 0, 2, 0] and order == [2, 0, 1, 3] and info == [4, 3, 2]


@pytest.mark.parametrize("new,old,kw", [
    ([100], [100], dict(old_block=16)),                        # more positions with a smaller block,
    ([100], [100], dict(old_stride=8)),                        # or a smaller stride,
    ([100, 1000], [100, 500], dict(old_block=16)),             # also where the last sequence has room
])
def test_a_cache_of_another_geometry_is_refused(new, old, kw):
    """Its positions do not fit into the new one: copying them would write past the sequence's rows."""
    rc, _, _ = _plan(new, old, **kw)
    assert rc == -18 and b"sequence 0" in _lib.lib().nsa_last_error()


def test_a_shorter_sequence_is_refused():
    assert _plan([40, 30], [40, 31])[0] == -17
