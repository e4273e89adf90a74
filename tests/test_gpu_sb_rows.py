"""Superblock row generation at the edges of its launch: more terms than a warp holds at once, rows
past each buffer size, and the two-pass build of a superblock whose generated elements exceed the
scratch of the single pass.  All bit for bit the oracle's."""
import numpy as np
import pytest

from dmrg_c_gb300 import sb_models, workloads

pytestmark = pytest.mark.gpu


def _repeated(m, k, keep=None):
    """The term list k times over (every target k times, summed in generation order)."""
    terms = [(t[0], t[1], t[2], t[3], t[4] * (1.0 + 0.25 * i), t[5], t[6]) for i in range(k) for t in m.terms]
    return sb_models.SBModel(m.n, m.dim_LL, m.dim_RR, m.d, m.LL, m.LR, m.RR, m.RL, m.inv, m.ops, terms[:keep], m.ele)


def _generated(m):
    """Generated elements of every row."""
    st, g = (m.LL, m.LR, m.RR, m.RL), np.zeros(m.n, np.int64)
    for p1, p2, o1, o2, *_ in m.terms:
        c = np.diff(m.ops[o1].row)[st[p1]]
        g += c * np.diff(m.ops[o2].row)[st[p2]] if p2 >= 0 else c
    return g


def _check(gpu, oracle, m):
    for a, b in zip(gpu.SuperblockCRS(m).download(), oracle.sb_build(m)):
        assert np.array_equal(a.view(np.int64) if a.dtype == np.float64 else a, b.view(np.int64) if b.dtype == np.float64 else b)


@pytest.mark.parametrize("keep", [1, 4, 31, 32, 33, 64, 65])
def test_rows_term_counts(gpu, oracle, keep):
    _check(gpu, oracle, _repeated(sb_models.small_hubbard_model(True), 5, keep))


@pytest.mark.parametrize("k", [2, 8, 30, 55])
def test_rows_buffer_sizes(gpu, oracle, k):
    m = _repeated(sb_models.small_hubbard_model(False), k)
    assert _generated(m).max() < 4096
    _check(gpu, oracle, m)


def test_rows_two_pass(gpu, oracle):
    m = _repeated(workloads.hubbard_sb_model_m512(0, per_row=128), 4)
    assert 12 * int(np.sum(_generated(m) + 1)) > 2 << 30   # past the single pass' scratch
    _check(gpu, oracle, m)
