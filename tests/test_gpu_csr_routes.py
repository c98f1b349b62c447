"""Systems whose size and number of entries would allow prgpu_cg_csr's streamed product but whose rows it is slow on
go to a thread per row, which nz = 0 picks by itself: the same solution bit for bit, where the streamed product's,
whose FP64 sums run in another order, is made to differ."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (1 << 17) + 45


def _system(kind):
    """Rows as (lengths, columns of entry j of each row); the first entry is the diagonal."""
    rng = np.random.default_rng(5)
    row = np.arange(N)
    near = lambda w: (row[:, None] + np.arange(w)) % N                          # noqa: E731
    if kind == "scattered":             # columns anywhere
        col = np.concatenate([row[:, None], rng.integers(0, N, (N, 19))], 1)
        return np.full(N, 20), col, 20 * N
    if kind == "mostly_scattered":      # two rows in three
        col = near(24)
        col[row % 96 < 64, 1:] = rng.integers(0, N, (int((row % 96 < 64).sum()), 23))
        return np.full(N, 24), col, 24 * N
    if kind == "one_bank":              # every row starts in the same bank of shared memory, columns 3,000 around
        return np.full(N, 32), (row[:, None] + np.concatenate([[[0]] * N, rng.integers(0, 3000, (N, 31))], 1)) % N, 32 * N
    if kind == "uneven":                # rows of 1 to 199 entries
        return rng.integers(1, 200, N), near(199), 100 * N
    if kind == "near":
        return np.full(N, 27), near(27), 27 * N
    if kind == "long":
        return np.full(N, 161), near(161), 161 * N
    if kind == "wrong_nz":              # three entries a row, thirty claimed
        return np.full(N, 3), near(3), 30 * N


def _solve(kind):
    import torch
    import poissonrecon_gpu_gb300 as pg
    L = pg._lib()
    length, col, nz = _system(kind)
    keep = np.arange(col.shape[1]) < length[:, None]
    ptr = np.zeros(N + 1, np.int32)
    ptr[1:] = np.cumsum(length)
    # q = A p = +-p, so that p.q cancels to the rounding of its FP64 sums: the first step's length, and with it x, is
    # their order's
    half = N // 2
    val = np.zeros(col.shape, np.float32)
    val[:, 0] = np.where(np.arange(N) < half, 1, -1)
    rng = np.random.default_rng(2)
    b = np.zeros(N, np.float32)
    b[:half] = rng.standard_normal(half) * np.exp2(rng.uniform(-25, 25, half))
    b[half:2 * half] = rng.permutation(b[:half])
    t = [torch.from_numpy(a).cuda() for a in (ptr, col[keep].astype(np.int32), val[keep], b)]
    out = []
    for entries in (nz, 0):
        x = torch.zeros(N, device="cuda")
        it = ctypes.c_int32(0)
        L.prgpu_cg_csr(N, entries, *[a.data_ptr() for a in t], x.data_ptr(), 0.0, 1, ctypes.byref(it), None)
        assert it.value == 1
        out.append(x.cpu().numpy())
    return np.array_equal(out[0], out[1], equal_nan=True)


@pytest.mark.parametrize("kind", ["scattered", "mostly_scattered", "one_bank", "uneven", "long", "wrong_nz"])
def test_declined_systems_take_a_thread_per_row(lib_built, kind):
    assert _solve(kind)


def test_near_columns_are_streamed(lib_built):
    assert not _solve("near")
