"""CRS_CRS_CCS_PRODUCT where its shortcuts could go wrong: lines whose supports touch, overlap or lie
apart, unsorted and repeated indices, empty lines, and infinities (a zero times an infinity is not
zero, so nothing may be skipped).  Bit for bit the oracle's."""
import numpy as np
import pytest

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu


def _lines(rng, n, dim, blocks, repeat, empty, shuffle):
    ptr, idx = [0], []
    for l in range(n):
        b = l * blocks // n
        lo, hi = b * dim // blocks, (b + 1) * dim // blocks
        k = 0 if rng.random() < empty else int(rng.integers(1, hi - lo + 1))
        c = rng.choice(np.arange(lo, hi), size=k, replace=False)
        c = np.concatenate([c, rng.choice(c, size=k // 2)]) if repeat and k else c
        c = rng.permutation(c) if shuffle else np.sort(c, kind="stable")
        idx += c.tolist()
        ptr.append(len(idx))
    return np.array(ptr), np.array(idx, np.int32), rng.standard_normal(len(idx))


def _check(gpu, oracle, M1, M2, M3, r2, c3, r1):
    with np.errstate(all="ignore"):
        want = oracle.crs_crs_ccs(M1, M2, M3)
    got = oracle.call_crs_crs_ccs(gpu.load(), M1, M2, M3, max(r2 * c3, 1), max(r1 * c3, 1))
    for a, b in zip(got[:6], want):
        a, b = np.asarray(a), np.asarray(b)
        assert a.shape == b.shape
        if b.dtype == np.float64:
            assert np.array_equal(a.astype(np.float64).view(np.int64), b.view(np.int64))
        else:
            assert np.array_equal(a, b)


@pytest.mark.parametrize("r1,r2,r3,c3", [(1, 1, 1, 1), (7, 33, 40, 9), (31, 256, 257, 33), (64, 300, 513, 65)])
@pytest.mark.parametrize("blocks,repeat,shuffle", [(1, False, False), (5, False, False), (5, True, True)])
def test_supports(gpu, oracle, r1, r2, r3, c3, blocks, repeat, shuffle):
    rng = np.random.default_rng([r1, r2, blocks, repeat])
    nb = min(blocks, r1, r2, r3, c3)
    M1 = abi.Crs(*_lines(rng, r1, r2, nb, repeat, 0.1, shuffle), n=r1, ncol=r2)
    M2 = abi.Crs(*_lines(rng, r2, r3, nb, repeat, 0.1, shuffle), n=r2, ncol=r3)
    M3 = abi.Ccs(*_lines(rng, c3, r3, nb, repeat, 0.1, shuffle), r3, c3)
    _check(gpu, oracle, M1, M2, M3, r2, c3, r1)


@pytest.mark.parametrize("where", ["m1", "m2", "m3", "overflow"])
def test_infinities(gpu, oracle, where):
    rng = np.random.default_rng(5)
    r1, r2, r3, c3 = 20, 60, 70, 20
    a, b, c = _lines(rng, r1, r2, 4, False, 0.0, False), _lines(rng, r2, r3, 4, False, 0.0, False), _lines(rng, c3, r3, 4, False, 0.0, False)
    if where == "overflow":   # finite operands, an infinite intermediate
        b[2][::3] = 1e200
        c[2][::2] = 1e200
    else:
        {"m1": a, "m2": b, "m3": c}[where][2][3] = np.inf
    _check(gpu, oracle, abi.Crs(*a, n=r1, ncol=r2), abi.Crs(*b, n=r2, ncol=r3), abi.Ccs(*c, r3, c3), r2, c3, r1)
