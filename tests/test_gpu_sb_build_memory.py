"""A superblock build on a device with room for the single pass' scratch or for the result but not for
both: it falls back to the two passes and gives the CRS it gives with room for both."""
import numpy as np
import pytest

from dmrg_c_gb300 import workloads

pytestmark = pytest.mark.gpu


def _generated(m):
    st, g = (m.LL, m.LR, m.RR, m.RL), np.zeros(m.n, np.int64)
    for p1, p2, o1, o2, *_ in m.terms:
        c = np.diff(m.ops[o1].row)[st[p1]]
        g += c * np.diff(m.ops[o2].row)[st[p2]] if p2 >= 0 else c
    return g


def _same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x.view(np.int64) if x.dtype == np.float64 else x, y.view(np.int64) if y.dtype == np.float64 else y)


def test_room_for_scratch_or_result(gpu):
    import torch

    m = workloads.hubbard_sb_model_m512(0, per_row=128)
    want = gpu.SuperblockCRS(m).download()
    scratch, result = 12 * int(np.sum(_generated(m) + 1)), 12 * len(want[1])
    assert scratch < 2 << 30 and result > 64 << 20
    assert gpu.load().dg_release_pool() == 0
    # what the build holds beside the two, and the pool's rounding
    inputs = 64 * m.n + 4 * len(m.inv) + (32 << 20)
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - (inputs + scratch + result // 2), dtype=torch.uint8, device="cuda")
    try:
        _same(gpu.SuperblockCRS(m).download(), want)
    finally:
        del hold
        torch.cuda.empty_cache()
