"""The range of operator scales FP64 Lanczos takes.  Multiplying an operator by a power of two multiplies
every number the recurrence forms by one, so the eigenvalue scales, and the vector and the step counts stay,
bit for bit, as far as the squared norms <Hv,Hv> stay inside the double range."""
import numpy as np
import pytest
import scipy.sparse as sp

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu

SCALES = [-480, -400, -300, 300, 340, 480]


def _operator(zero_diagonal):
    rng = np.random.default_rng(11)
    n = 1500
    A = sp.random(n, n, density=8.0 / n, random_state=rng, data_rvs=rng.standard_normal)
    A = (A + A.T).tolil()
    A.setdiag(0.0 if zero_diagonal else rng.uniform(-1, 1, n))
    A[3, 7] = A[7, 3] = 12.0   # a gap: eigenvalues near +-12
    A = A.tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    return A


@pytest.mark.parametrize("restart", [False, True])
@pytest.mark.parametrize("zero_diagonal", [False, True])
def test_power_of_two_scales(gpu, zero_diagonal, restart):
    A = _operator(zero_diagonal)
    rng = np.random.default_rng(2)
    guess = rng.standard_normal(A.shape[0])
    if zero_diagonal:   # and a first alpha of zero: the operator has no element inside either half
        half = np.arange(A.shape[0]) % 2
        B = A.tocoo()
        keep = half[B.row] != half[B.col]
        A = sp.csr_matrix((B.data[keep], (B.row[keep], B.col[keep])), shape=A.shape).tolil()
        A[2, 7] = A[7, 2] = 12.0
        A = A.tocsr()
        A.sort_indices()
        guess[half == 1] = 0.0
    acc = 1e-13

    def solve(k):
        m = gpu.DeviceMatrix(abi.Crs.from_scipy(sp.csr_matrix((np.ldexp(A.data, k), A.indices, A.indptr), shape=A.shape)))
        p = gpu.default_params(dense_below=0, lanczos_acc=np.ldexp(acc, k), lanczos_block_step=30 if restart else 800)
        return gpu.ground_state(m, p, guess=guess, lanczos_only=True)

    v0, i0 = solve(0)
    exact = np.linalg.eigvalsh(A.toarray())[0]
    assert i0.dense == 0 and abs(i0.eig_val - exact) <= 1e-11 * abs(exact)
    for k in SCALES:
        v, i = solve(k)
        assert i.converged and i.lanczos_steps == i0.lanczos_steps, k
        assert i.eig_val == np.ldexp(i0.eig_val, k), k
        assert np.array_equal(v, v0), k
