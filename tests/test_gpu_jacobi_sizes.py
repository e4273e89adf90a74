"""Density-block eigensolver at the edges of its launch rules: one block of n pairs for every n where
the cluster size, the threads, who forms the rotations or the memory the rows live in changes, and
mixed sizes together.  Checked against 64-bit numpy: spectrum, orthonormality and eigen-equation
within n * 2^-52 of the norm times a small factor (Jacobi's error bound: a few roundings a sweep,
at most 20 sweeps)."""
import ctypes as C

import numpy as np
import pytest

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu


def _truncate(gpu, sizes, Q, keep, seed):
    """DMRG_GET_SYSTEM_INFO_Q1 on blocks of the given sizes (label g: sizes[g] block states, each with
    the same Q states of the other block)."""
    rng = np.random.default_rng(seed)
    dim_LL, dim_RR = int(np.sum(sizes)), len(sizes) * Q
    label = np.repeat(np.arange(len(sizes)), sizes)
    LL = np.repeat(np.arange(dim_LL), Q)
    RR = (label[:, None] * Q + np.arange(Q)[None, :]).ravel()
    n = len(LL)
    X = [rng.standard_normal((s, Q)) * 0.7 ** np.arange(s)[:, None] for s in sizes]
    v = np.concatenate([x.ravel() for x in X])
    v /= np.linalg.norm(v)
    zero = np.zeros(n, np.int16)
    st = [LL.astype(np.int16), zero, RR.astype(np.int16), zero]
    inv = -np.ones(dim_LL * dim_RR, np.int32)
    inv[LL.astype(np.int64) * dim_RR + RR] = np.arange(n)
    pairs = [np.arange(dim_LL, dtype=np.int16), np.zeros(dim_LL, np.int16)]
    cnt, lab = np.full(dim_LL, Q, np.int32), label.astype(np.int32)
    B = abi.DMRG_BASIS(LL_LLLRRRRL=abi.ptr(st[0], C.c_short), LR_LLLRRRRL=abi.ptr(st[1], C.c_short),
                       RR_LLLRRRRL=abi.ptr(st[2], C.c_short), RL_LLLRRRRL=abi.ptr(st[3], C.c_short),
                       Inv_LLLRRRRL=abi.ptr(inv, C.c_int), dim_LLLRRRRL=n, dim_LL=dim_LL, dim_RR=dim_RR, dim_onsite=1,
                       LL_LLLR=abi.ptr(pairs[0], C.c_short), LR_LLLR=abi.ptr(pairs[1], C.c_short), dim_LLLR=dim_LL,
                       Sum_LLLR=abi.ptr(cnt, C.c_int))
    T = abi.DMRG_TIME()
    S = gpu.load().DMRG_GET_SYSTEM_INFO_Q1(abi.ptr(lab, C.c_int), C.byref(B), abi.ptr(v, C.c_double), keep, 1, C.byref(T)).contents
    k, M = S.dim_renorm, S.Trans_Matrix.contents
    w = np.array(S.Val_DM_Dist[:dim_LL])
    D = np.zeros((dim_LL, k))
    for j in range(k):
        D[M.Row[M.Col[j]:M.Col[j + 1]], j] = M.Val[M.Col[j]:M.Col[j + 1]]
    X, at = [], 0
    for s in sizes:
        X.append(v[at:at + s * Q].reshape(s, Q))
        at += s * Q
    return w, D, X


@pytest.mark.parametrize("sizes", [[1], [2], [3], [8], [31], [63], [64], [65], [111], [112], [113], [127], [260], [261], [345],
                                   [360], [361], [368], [369], [400], [40, 3, 1, 17], [113, 112, 64, 5], [369, 120, 30]])
def test_block_sizes(gpu, sizes):
    n, Q = max(sizes), max(max(sizes) // 2, 3)
    w, D, X = _truncate(gpu, sizes, Q, max(1, sum(sizes) // 3), 11 + n)
    rho = np.zeros((sum(sizes),) * 2)
    at = 0
    for x in X:
        rho[at:at + len(x), at:at + len(x)] = x @ x.T
        at += len(x)
    norm = np.linalg.norm(rho, 2)
    tol = 20 * n * 2.0 ** -52
    want = np.sort(np.concatenate([np.linalg.eigvalsh(x @ x.T) for x in X]))[::-1]
    assert np.max(np.abs(w - want)) <= tol * norm
    assert np.max(np.abs(D.T @ D - np.eye(D.shape[1]))) <= tol
    kept = np.einsum("ij,ij->j", D, rho @ D)
    assert np.max(np.abs(rho @ D - D * kept)) <= tol * norm
    assert np.max(np.abs(np.sort(kept)[::-1] - want[:D.shape[1]])) <= tol * norm
