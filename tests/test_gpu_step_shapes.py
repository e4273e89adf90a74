"""Lanczos and CG at the sizes where their vector kernels change shape (threads a block, blocks a SM),
one row either side of each, and at one row and one block.  A tridiagonal matrix with one deep site:
its lowest eigenvalue to 1e-12 against LAPACK's bisection, and CG to its stopping residual."""
import numpy as np
import pytest
import scipy.linalg as sl

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu

SMS = 152
SIZES = [2, 31, 255, 256, 257, 1000, SMS * 512 - 1, SMS * 512, SMS * 512 + 1, SMS * 2048, SMS * 2048 + 1]


def _tridiagonal(n, seed):
    rng = np.random.default_rng(seed)
    d = 2.0 + rng.uniform(0, 1, n)
    d[n // 3] = -3.0
    e = -0.3 * rng.uniform(0.5, 1, n - 1)
    row = np.concatenate([[0], np.cumsum(np.r_[1, np.full(n - 1, 2)])]).astype(np.int64)   # lower triangle, diagonal last
    col = np.empty(2 * n - 1, np.int32)
    val = np.empty(2 * n - 1)
    col[0], val[0] = 0, d[0]
    col[1::2], val[1::2] = np.arange(n - 1), e
    col[2::2], val[2::2] = np.arange(1, n), d[1:]
    return d, e, abi.Crs(row, col, val, n=n)


@pytest.mark.parametrize("n", SIZES)
def test_lanczos_and_cg(gpu, n):
    d, e, A = _tridiagonal(n, n)
    m = gpu.DeviceMatrix(A, gpu.DG_STORE_LOWER_DIAG_LAST)
    p = gpu.default_params(seed=3, dense_below=0)
    v, info = gpu.ground_state(m, p)
    want = sl.eigh_tridiagonal(d, e, select="i", select_range=(0, 0))[0][0] if n > 2 else np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))[0]
    assert abs(info.eig_val - want) <= 1e-12 * abs(want)

    def product(x):
        y = d * x
        y[:-1] += e * x[1:]
        y[1:] += e * x[:-1]
        return y

    assert np.linalg.norm(product(v) - want * v) <= 1e-9
    b = np.random.default_rng(7).standard_normal(n)
    x = np.ones(n)
    sigma, acc = 4.0, 1e-16 * n
    rc, it = gpu.linear_solve(m, b, x, sigma=sigma, acc=acc, max_step=200)
    assert rc == 0 and it < 200
    # the recurrence's residual and the true one differ by a few roundings of ||A|| ||x|| an iteration
    assert np.linalg.norm(product(x) + sigma * x - b) <= np.sqrt(acc) + it * 8 * np.linalg.norm(x) * 2.0 ** -52 * 10
