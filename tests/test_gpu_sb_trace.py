"""Expectation values through the reduced density matrices at the sizes where their kernels can go
wrong: rows with more needed entries than a warp collects at once, sums shorter than the lanes
that share them and past a full turn of them, one site state, each position alone (only that half's
entries are formed), and a weight vector that is not v."""
import numpy as np
import pytest

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (2, 3, 1), (70, 3, 1), (3, 70, 1), (40, 33, 1), (5, 9, 2), (33, 16, 2), (65, 8, 3), (17, 130, 2), (21, 11, 4)]


def _operator(rng, n):
    """A random operator with empty rows and one full row."""
    m = rng.standard_normal((n, n)) * (rng.random((n, n)) < 0.4)
    m[rng.integers(n)] = 0.0
    m[rng.integers(n)] = rng.standard_normal(n)
    cols = [np.flatnonzero(r) for r in m]
    return m, abi.Crs(np.concatenate([[0], np.cumsum([len(c) for c in cols])]), np.concatenate(cols).astype(np.int32),
                      np.concatenate([r[c] for r, c in zip(m, cols)]))


def _dense(basis, x, d):
    t = np.zeros((basis.dim_LL, d, basis.dim_RR, d))
    ll, lr, rr, rl, _ = basis.download()
    t[ll, lr, rr, rl] = x
    return t, (ll, lr, rr, rl)


@pytest.mark.parametrize("blocks", [1, 3])
@pytest.mark.parametrize("dl,dr,d", SIZES)
def test_traces_at_edge_sizes(gpu, dl, dr, d, blocks):
    rng = np.random.default_rng(100 * dl + dr + blocks)
    q_l, q_r = np.arange(dl) % blocks, -(np.arange(dr) % blocks)
    basis = gpu.SuperblockBasis(dl, dr, d, q_l, q_r, np.zeros(d, np.int32), 0)
    dims = (dl, d, dr, d)
    mats, crs = zip(*[_operator(rng, n) for n in dims])
    ops = gpu.BlockOperators(list(crs), list(dims))
    v, w = rng.standard_normal((2, basis.n))
    tv, at = _dense(basis, v, d)
    out = "abcd"
    for pos, only in [(p, True) for p in range(4)] + [(None, False)]:
        for second in (None, w):
            terms = [(p, p, 0, int(second is not None)) for p in range(4) if not only or p == pos]
            got = gpu.sb_expect(basis, basis, ops, terms, v, v, second)
            weight = v if second is None else second
            for g, (p, *_) in zip(got, terms):
                sub = f"{out[p]}x,{out.replace(out[p], 'x')}->{out}"
                want = np.dot(weight, np.einsum(sub, mats[p], tv)[at])
                size = np.dot(np.abs(weight), np.einsum(sub, np.abs(mats[p]), np.abs(tv))[at])
                # every product passes through fewer roundings than there are states, plus the trees
                assert abs(g - want) <= (basis.n + 64) * 2.0 ** -53 * size, (p, g, want)
