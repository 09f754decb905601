"""A pointer handed to the library keeps its array: an array made for the
call alone (the weir parameters of a batch) is read by the call, not by whoever
is given its memory next."""
import gc
import weakref

import numpy as np

from braids_hkt_gb300.solver import _ptr


def test_pointer_holds_a_temporary():
    a = np.arange(240.0)
    alive, address = weakref.ref(a), a.ctypes.data
    p = _ptr(a)
    del a
    gc.collect()
    assert alive() is not None and p.value == address
    del p
    assert alive() is None
    assert _ptr(None) is None
