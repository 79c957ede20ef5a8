"""Edge counts that no device holds are refused before any memory is asked for
or read: the sizes that follow from them must not wrap."""
import ctypes

import numpy as np
import pytest


@pytest.mark.parametrize("n,flags,status", [
    (1 << 60, 0, -3), ((1 << 60) - 1, 4, -3), (1 << 59, 1, -3), ((1 << 59) - 7, 5, -3), ((1 << 60) + 1, 0, -1),
    ((1 << 59) + 1, 1, -1), (1 << 63, 0, -1),
])
def test_edge_counts_past_every_device(gw, n, flags, status):
    L = gw.load()
    ids = np.array([0, 1], np.uint32)
    p = ctypes.c_void_p(ids.ctypes.data)
    beg, csr, ne, nv = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_uint64(), ctypes.c_uint32()
    assert L.gw_edges_csr(p, p, n, 2, flags, ctypes.byref(beg), ctypes.byref(csr), ctypes.byref(ne),
                          ctypes.byref(nv)) == status
    assert not beg.value and not csr.value
