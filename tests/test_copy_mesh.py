"""prgpu_copy_mesh: every byte and no other, around the size from which several threads share the copy and at
destinations off the page boundaries that the parts are cut at."""
import ctypes

import numpy as np
import pytest

WIDE = 16 << 20


@pytest.mark.parametrize("nv,nt,shift", [(0, 0, 0), (1, 2, 3), (WIDE // 12 - 1, 1, 1), (WIDE // 12 + 1, WIDE // 12, 0),
                                         (WIDE // 12 + 7, 2 * WIDE // 12 + 5, 1021), (40_000_003 // 12, 3, 524_287)])
def test_copy_mesh(lib_built, nv, nt, shift):
    import poissonrecon_gpu_gb300 as pg
    rng = np.random.default_rng(nv + nt)
    v = rng.random(3 * nv, dtype=np.float32)
    f = rng.integers(0, 1 << 30, 3 * nt, dtype=np.int32)
    m = pg.Mesh(nv, nt, v.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), f.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)))
    dv = np.full(3 * nv + 2 * shift + 2, -1, np.float32)
    df = np.full(3 * nt + 2 * shift + 2, -1, np.int32)
    assert pg._lib().prgpu_copy_mesh(ctypes.byref(m), dv[shift:].ctypes.data, df[shift:].ctypes.data) == 0
    for d, s in ((dv, v), (df, f)):
        assert np.array_equal(d[shift:shift + len(s)], s)
        assert np.all(d[:shift] == -1) and np.all(d[shift + len(s):] == -1)


def test_copy_mesh_refuses_null(lib_built):
    import poissonrecon_gpu_gb300 as pg
    assert pg._lib().prgpu_copy_mesh(ctypes.byref(pg.Mesh(1, 0)), None, None) == 1
    assert pg._lib().prgpu_copy_mesh(None, None, None) == 1
