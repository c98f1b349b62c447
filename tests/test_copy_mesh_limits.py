"""prgpu_copy_mesh on meshes that cannot be: a negative count is refused before anything is copied."""
import ctypes

import numpy as np
import pytest


@pytest.mark.parametrize("nv,nt", [(-1, 0), (0, -1), (-(1 << 40), 1), (2, -3)])
def test_negative_counts_are_refused(lib_built, nv, nt):
    import poissonrecon_gpu_gb300 as pg
    v, f = np.ones(6, np.float32), np.ones(6, np.int32)
    dv, df = np.zeros(6, np.float32), np.zeros(6, np.int32)
    m = pg.Mesh(nv, nt, v.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), f.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)))
    assert pg._lib().prgpu_copy_mesh(ctypes.byref(m), dv.ctypes.data, df.ctypes.data) == 1
    assert not dv.any() and not df.any()
