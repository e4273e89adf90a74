"""Expansion of a lower triangle to full rows and the sliced-ELL fill at the edges of their kernels: upper
parts at and past each register sort's size and past the largest, matrices with more rows than the
32-bit sort keys hold, every sorting window, and rows shorter and longer than a fill tile.  Values are
small integers, so that every product is exact in FP64 and in FP32 and compared bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu

PARTS = [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300, 17, 15, 16]


def _lower(rng, n, copies):
    """Lower triangle, diagonal last: columns of every upper part's length, at random rows below."""
    r, c = [np.arange(n)], [np.arange(n)]
    top = n - max(PARTS) - 1
    for col, m in zip(rng.choice(top, copies * len(PARTS), replace=False), copies * PARTS):
        r.append(col + 1 + rng.choice(min(n - col - 1, 1 << 20), m, replace=False))
        c.append(np.full(m, col))
    r, c = np.concatenate(r), np.concatenate(c)
    v = rng.integers(1, 9, len(r)).astype(np.float64)
    return sp.csr_matrix((v, (r, c)), shape=(n, n))


def _stored(lengths, window):
    n = -len(lengths) % 2048
    lens = np.concatenate([lengths, np.zeros(n, np.int64)])
    lens = -np.sort(-lens.reshape(-1, window), axis=1) if window > 32 else lens
    return int(32 * lens.reshape(-1, 32).max(axis=1).sum())


@pytest.mark.parametrize("n,copies", [(331, 1), (2049, 3), (5000, 40), ((1 << 24) + 70, 2)])
def test_expansion_and_fill(gpu, monkeypatch, n, copies):
    monkeypatch.setenv("DG_SELL_DELTAS", "0")   # the large one would take the delta stream's own fill
    rng = np.random.default_rng(n + copies)
    low = _lower(rng, n, min(copies, (n - 301) // len(PARTS)))
    full = (low + sp.tril(low, -1).T).tocsr()
    full.sort_indices()
    m = gpu.DeviceMatrix(abi.Crs.from_scipy(low), gpu.DG_STORE_LOWER_DIAG_LAST, gpu.DG_VALUES_BOTH)
    row, col, val = m.download()
    assert np.array_equal(row, full.indptr) and np.array_equal(col, full.indices) and np.array_equal(val, full.data)
    x = rng.integers(-4, 5, n).astype(np.float64)
    want = full @ x
    for window in (2048,) if n > 1 << 20 else (2048, 32, 64, 512, 1024):
        m.set_sell_window(window)
        assert m.format() == (gpu.DG_FORMAT_SELL, _stored(np.diff(full.indptr), window))
        assert np.array_equal(m.spmv(x), want), window
        assert np.array_equal(m.spmv_f32(x.astype(np.float32)), want.astype(np.float32)), window
