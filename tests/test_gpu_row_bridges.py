"""The check for the 16-bit column stream on rows of a few elements, several rows a warp: row lengths around
the lanes a row has, counts of bridges, and a decreasing column found wherever in its row it is."""
import numpy as np
import pytest

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu

BRIDGE = 65535


def _rows(n, swap=None):
    rng = np.random.default_rng(n)
    lengths = rng.integers(0, 20, n)
    lengths[-3:] = (9, 17, 18)   # the last warp's rows
    row = np.concatenate([[0], np.cumsum(lengths)])
    k = np.arange(row[-1]) - np.repeat(row[:-1], lengths)
    first = np.repeat(rng.integers(0, n - 190_000, n), lengths)
    jump = np.repeat((rng.random(n) < 0.04) * rng.integers(60_000, 180_000, n), lengths)
    jump_at = np.repeat(rng.integers(1, 20, n), lengths)
    col = first + 3 * k + jump * (k >= jump_at)
    col[row[-3]:] = np.minimum(col[row[-3]:], n - 1)
    if swap is not None:   # columns swap - 1 and swap of the last row decrease
        i = row[-2] + swap
        col[i - 1], col[i] = col[i], col[i - 1]
    return row, col.astype(np.int32)


def _bridges(row, col):
    gap = np.diff(col.astype(np.int64))
    inside = np.ones(len(gap), bool)
    starts = row[1:-1]
    inside[starts[(starts > 0) & (starts < len(col))] - 1] = False
    return int(np.maximum(0, (gap[inside] - 1) // BRIDGE).sum())


@pytest.mark.parametrize("n", [200_000, 200_001, 200_002, 200_003])
def test_bridge_counts(gpu, monkeypatch, n):
    monkeypatch.setenv("DG_SELL_DELTAS", "1")
    row, col = _rows(n)
    want = _bridges(row, col)
    assert 0 < want <= row[-1] // 32
    m = gpu.DeviceMatrix(abi.Crs(row, col, np.ones(len(col))), gpu.DG_STORE_FULL, gpu.DG_VALUES_BOTH)
    present, bridges = m.sell_deltas()
    assert present and bridges == want


@pytest.mark.parametrize("swap", [1, 7, 8, 9, 16, 17])
def test_decreasing_columns(gpu, monkeypatch, swap):
    monkeypatch.setenv("DG_SELL_DELTAS", "1")
    row, col = _rows(200_001, swap)
    m = gpu.DeviceMatrix(abi.Crs(row, col, np.ones(len(col))), gpu.DG_STORE_FULL, gpu.DG_VALUES_BOTH)
    assert not m.sell_deltas()[0]
