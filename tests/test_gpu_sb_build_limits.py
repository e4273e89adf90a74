"""Superblock builds side by side on several threads, of rows that need different amounts of shared memory:
each gives the CRS it gives alone."""
import threading

import numpy as np
import pytest

from dmrg_c_gb300 import sb_models

pytestmark = pytest.mark.gpu


def _repeated(m, k):
    terms = [(t[0], t[1], t[2], t[3], t[4] * (1.0 + 0.25 * i), t[5], t[6]) for i in range(k) for t in m.terms]
    return sb_models.SBModel(m.n, m.dim_LL, m.dim_RR, m.d, m.LL, m.LR, m.RR, m.RL, m.inv, m.ops, terms, m.ele)


def _generated(m):
    st, g = (m.LL, m.LR, m.RR, m.RL), np.zeros(m.n, np.int64)
    for p1, p2, o1, o2, *_ in m.terms:
        c = np.diff(m.ops[o1].row)[st[p1]]
        g += c * np.diff(m.ops[o2].row)[st[p2]] if p2 >= 0 else c
    return g


def _same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x.view(np.int64) if x.dtype == np.float64 else x, y.view(np.int64) if y.dtype == np.float64 else y)


def test_builds_at_once(gpu):
    small = sb_models.small_hubbard_model(False)
    models = [_repeated(small, k) for k in (1, 8, 30, 55)]
    assert _generated(models[0]).max() < 64 and _generated(models[-1]).max() > 512   # 4 KB a block against 64
    want = [gpu.SuperblockCRS(m).download() for m in models]
    errors = []

    def build(k):
        try:
            for _ in range(60):
                _same(gpu.SuperblockCRS(models[k]).download(), want[k])
        except Exception as e:   # noqa: BLE001 (raised below, on the test's own thread)
            errors.append(e)

    threads = [threading.Thread(target=build, args=(k % len(models),)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
