"""The dense path's cluster step at the edges of its shapes: one state, each cluster size and one row
either side of it, the largest system and one past it (the kernel-per-phase form), Krylov spaces
longer than a coefficient chunk and than the part of the basis kept in shared memory.  Energies to
1e-12 and vectors to 1e-9 against numpy's dense eigensolver (a random symmetric matrix with one low
state: a gap of order one)."""
import numpy as np
import pytest
import scipy.sparse as sp

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu


def _matrix(n, per_row, seed):
    rng = np.random.default_rng(seed)
    A = sp.random(n, n, density=min(1.0, per_row / (2 * n)), random_state=rng, data_rvs=rng.standard_normal)
    A = (A + A.T + sp.diags(rng.uniform(0, 2, n))).tolil()
    A[n // 2, n // 2] = -3.0 - 0.5 * per_row
    return A.tocsr()


@pytest.mark.parametrize("n,per_row", [(1, 1), (2, 2), (3, 2), (31, 4), (32, 4), (33, 4), (64, 6), (65, 6), (128, 8), (129, 40), (256, 8),
                                       (257, 8), (511, 8), (512, 30), (513, 8), (924, 7), (999, 60), (1023, 8), (1024, 8), (1025, 8)])
def test_dense_sizes(gpu, n, per_row):
    A = _matrix(n, per_row, n)
    m = gpu.DeviceMatrix(abi.Crs.from_scipy(A))
    v, info = gpu.ground_state(m, gpu.default_params(seed=2, dense_below=2000))
    w, V = np.linalg.eigh(A.toarray())
    assert info.dense == 1
    assert abs(info.eig_val - w[0]) <= 1e-12 * max(1.0, abs(w[0]))
    assert abs(abs(v @ V[:, 0]) - 1.0) <= 1e-9


@pytest.mark.parametrize("n", [300, 999])
def test_long_krylov_space(gpu, n):
    """Levels that crowd at the bottom of the spectrum: the Ritz vector needs most of the space (more
    than a chunk of 128 coefficients, and at 999 states more vectors than the shared memory keeps)."""
    A = sp.diags([np.linspace(0.0, 1.0, n) ** 2], [0]).tocsr()
    m = gpu.DeviceMatrix(abi.Crs.from_scipy(A))
    v, info = gpu.ground_state(m, gpu.default_params(seed=2))
    w, V = np.linalg.eigh(A.toarray())
    assert info.dense == 1 and info.lanczos_steps > 140
    assert abs(info.eig_val - w[0]) <= 1e-12
    assert np.linalg.norm(A @ v - w[0] * v) <= 1e-9
