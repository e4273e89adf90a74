"""Conjugate gradients of small systems, which run as one kernel on one thread-block cluster: systems of
one CTA and of sixteen, rows shorter and longer than the lanes that share one, the largest system the
form takes in each of its limits and the first past it, solves that end inside a chunk of
iterations, on its last and in a later one, and the iteration limit; against conjugate gradients in NumPy."""
import numpy as np
import pytest
import scipy.sparse as sp

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu


def _system(rng, n, per_row, spread):
    """Symmetric, diagonally dominant (eigenvalues >= 1): spread makes the solve longer."""
    k = n * (per_row // 2)
    A = sp.csr_matrix((rng.uniform(-1, 1, k), (rng.integers(0, n, k), rng.integers(0, n, k))), shape=(n, n))
    A = (A + A.T).tocsr()
    A.setdiag(0.0)
    A = (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + np.linspace(1.0, spread, n))).tocsr()
    A.sort_indices()
    return A


def _cg(A, b, x, sigma, acc, max_step):
    x = x / np.linalg.norm(x)
    r = b - (A @ x + sigma * x)
    p, rr = r.copy(), r @ r
    for it in range(1, max_step):
        y = A @ p + sigma * p
        a = rr / (p @ y)
        x, r = x + a * p, r - a * y
        new = r @ r
        if new < acc:
            return x, it
        p, rr = r + new / rr * p, new
    return x, max_step


@pytest.mark.parametrize("n,per_row,spread", [(1, 0, 1), (2, 2, 2), (31, 4, 3), (33, 4, 50), (64, 20, 9), (513, 6, 400),
                                              (924, 8, 3000), (924, 70, 9), (924, 74, 9), (2049, 30, 9), (4096, 8, 900),
                                              (4097, 8, 900)])
def test_small_system(gpu, n, per_row, spread):
    rng = np.random.default_rng(n + per_row)
    A = _system(rng, n, per_row, float(spread))
    m = gpu.DeviceMatrix(abi.Crs.from_scipy(A))
    b, x0, norm = rng.standard_normal(n), rng.standard_normal(n), abs(A).sum(axis=1).max()
    for sigma in (0.0, 0.625):
        for acc, max_step in ((1e-4, 1000), (1e-20, 1000), (0.0, 8), (0.0, 33), (0.0, 34)):
            want, steps = _cg(A, b, x0, sigma, acc, max_step)
            x = x0.copy()
            rc, it = gpu.linear_solve(m, b, x, sigma=sigma, acc=acc, max_step=max_step)
            assert rc == (0 if steps < max_step else 4) or acc == 0.0
            if acc == 0.0:
                if n > 64:   # (a smaller system is solved exactly before the limit)
                    assert rc == 4 and it == max_step
                continue
            assert abs(it - steps) <= 1
            # the smallest eigenvalue is >= 1, so the error is at most the residual; the recurred residual
            # drifts from the true one by some roundings of H x an iteration
            drift = 16 * it * 2.0 ** -53 * (norm + sigma) * (np.abs(want).max() + 1.0) * np.sqrt(n)
            assert np.linalg.norm(b - (A @ x + sigma * x)) <= np.sqrt(acc) + drift
            assert np.linalg.norm(x - want) <= 2 * np.sqrt(acc) + 2 * drift
