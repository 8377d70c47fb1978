"""The work buffers of a batch's workers (CPU): a worker's default children per batch by its share of the device, 35 bytes
each.  However many workers, together they hold no more than 32 workers of 2^25 children, and a thread with a sixteenth of
the device or more takes 2^26."""
import ctypes as C

import pytest

from sincfeyn_b200 import sq


@pytest.mark.parametrize('workers', range(1, 33))
def test_workers_together_stay_within_the_bound(workers):
    L = sq.lib()
    L.sqb_share_children.argtypes, L.sqb_share_children.restype = [C.c_double], C.c_long
    L.sqb_set_mem_share.argtypes, L.sqb_mem_share.restype = [C.c_double], C.c_double
    L.sqb_set_mem_share(1.0/workers)
    n = L.sqb_share_children(L.sqb_mem_share())
    L.sqb_set_mem_share(1.0)
    assert n*workers <= 32 << 25
    assert n == (1 << 26 if workers <= 16 else 1 << 25)
