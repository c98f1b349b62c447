"""reconstruct_batch's arrays are made in a callback on the library's host threads: what goes wrong there reaches the
caller as it was raised (an interrupt, memory that ran out), and not as the status the library ends with."""
import ctypes

import numpy as np
import pytest


class _Library:
    """prgpu_reconstruct_batch_into of clouds of four vertices and two triangles; a refused cloud ends the call."""

    def prgpu_reconstruct_batch_into(self, ctx, xyz, nrm, offsets, depths, n, alloc, user, outs):
        for k in range(n):
            pv, pf = ctypes.c_void_p(), ctypes.c_void_p()
            if alloc(user, k, 4, 2, ctypes.pointer(pv), ctypes.pointer(pf)) or not pv.value:
                return 3
            ctypes.memset(pv.value, 0, 48)
            ctypes.memset(pf.value, 0, 24)
        return 0

    def prgpu_last_error(self):
        return b"host allocation failed"

    def prgpu_destroy(self, ctx):
        return 0


@pytest.fixture
def batch(monkeypatch):
    import poissonrecon_gpu_gb300 as pg
    monkeypatch.setattr(pg, "_lib", lambda L=_Library(): L)
    r = object.__new__(pg.Reconstructor)
    r._h = ctypes.c_void_p()
    clouds = [(np.zeros((5, 3), np.float32), np.ones((5, 3), np.float32))] * 3
    return lambda: r.reconstruct_batch(clouds)


def test_arrays_come_back(batch):
    assert [(v.shape, f.shape) for v, f in batch()] == [((4, 3), (2, 3))] * 3


@pytest.mark.parametrize("error", [MemoryError, KeyboardInterrupt])
def test_what_the_callback_raises_reaches_the_caller(batch, monkeypatch, error):
    empty, calls = np.empty, []

    def failing(shape, dtype=float):
        calls.append(shape)
        if len(calls) == 4:             # the second cloud's triangles
            raise error()
        return empty(shape, dtype)

    monkeypatch.setattr(np, "empty", failing)
    with pytest.raises(error):
        batch()
