"""prgpu_cg_csr's two products: a thread per row, and the streamed one of systems with many entries a row.

The number of entries passed picks the product (nz = 0: a thread per row), so the same system runs
through both."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _banded(n, width, rng, long_row=None, empty=()):
    """Strictly diagonally dominant, symmetric: off-diagonals -1 at +-1..+-width, rows of different lengths."""
    rows = np.arange(n)
    keep = rng.random((width, n)) < 0.9          # entry (i, i + k + 1) and its mirror
    r, c = [rows], [rows]
    for k in range(width):
        i = rows[: n - k - 1][keep[k, : n - k - 1]]
        r += [i, i + k + 1]
        c += [i + k + 1, i]
    if long_row is not None:                     # one row longer than several pieces
        j = np.arange(width + 1, n - long_row - 1, 7)[:5000] + long_row
        r += [np.full(len(j), long_row), j]
        c += [j, np.full(len(j), long_row)]
    r, c = np.concatenate(r), np.concatenate(c)
    drop = np.isin(r, empty) | np.isin(c, empty)
    r, c = r[~drop], c[~drop]
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    ptr = np.zeros(n + 1, np.int32)
    ptr[1:] = np.cumsum(np.bincount(r, minlength=n))
    deg = np.diff(ptr)
    val = np.where(r == c, 1.25 * deg[r], -1.0).astype(np.float32)
    return ptr, c.astype(np.int32), val


@pytest.mark.parametrize("n,width,shift,long_row,empty", [
    (1 << 17, 13, 0, None, ()),                  # the smallest streamed system
    ((1 << 17) + 31, 9, 0, 5, (0, 77, 78)),      # a remainder of rows, a row of 5,000 entries, empty rows
    (200_003, 12, 1, 123_456, ()),               # arrays off a 16-byte boundary
    (152 * 480 * 2 + 1, 20, 0, None, ()),        # one row more than two per thread
])
def test_streamed_product_agrees_with_a_thread_per_row(lib_built, n, width, shift, long_row, empty):
    import torch
    import poissonrecon_gpu_gb300 as pg
    L = pg._lib()
    rng = np.random.default_rng(n)
    ptr, col, val = _banded(n, width, rng, long_row, empty)
    b = rng.standard_normal(n).astype(np.float32)
    b[list(empty)] = 0.0
    tp = torch.from_numpy(ptr).cuda()
    tc = torch.from_numpy(np.concatenate([np.zeros(shift, np.int32), col])).cuda()[shift:]
    tv = torch.from_numpy(np.concatenate([np.zeros(shift, np.float32), val])).cuda()[shift:]
    tb = torch.from_numpy(b).cuda()
    out = []
    assert len(val) >= 16 * n
    for nz in (len(val), 0):
        x = torch.zeros(n, device="cuda")
        it = ctypes.c_int32(0)
        assert L.prgpu_cg_csr(n, nz, tp.data_ptr(), tc.data_ptr(), tv.data_ptr(), tb.data_ptr(), x.data_ptr(),
                              1e-5, 1000, ctypes.byref(it), None) == 0
        out.append((x.cpu().numpy().astype(np.float64), it.value))
    # the products are the same bit for bit; only the order of the FP64 sums differs
    assert abs(out[0][1] - out[1][1]) <= 1
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-5
