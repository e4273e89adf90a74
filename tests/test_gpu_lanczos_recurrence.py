"""The FP64 Lanczos step against the recurrence in NumPy, from the same start vector and stopped well before
convergence: the step at which two energies first differ by less than 1e-6, the energy and the Ritz
vector there, for one to eight warps a slice, for CSR rows and across a restart.

Both sides round each of the <= 80 steps once or a few times relative to ||H||, and ghosts of a converged pair
do not appear before 1e-8: 1e-12 ||H|| for the energy, and for the vector 1e-12 ||H|| over the distance
of the two lowest Ritz values."""
import numpy as np
import pytest
import scipy.sparse as sp

from dmrg_c_gb300 import abi, workloads

pytestmark = pytest.mark.gpu

ACC = 1e-6


def _random(n):
    rng = np.random.default_rng(n)
    A = sp.random(n, n, density=min(1.0, 30.0 / n), random_state=rng, data_rvs=rng.standard_normal)
    return (A + A.T + sp.diags(rng.uniform(-1, 1, n))).tocsr()


def _superblock():
    low = workloads.xxz_superblock_m64(0).explicit_lower()
    L = sp.csr_matrix((low.val, low.col, low.row), shape=(low.n, low.n))
    return (L + sp.tril(L, -1).T).tocsr()


def _lanczos(A, w, block):
    """Steps, energy, normalised Ritz vector and the gap of the last tridiagonal."""
    E, total = 1e15, 0
    while True:
        V, d, e = [w / np.linalg.norm(w)], [], []
        for b in range(block):
            y = A @ V[b]
            d.append(V[b] @ y)
            w = y - d[b] * V[b] - (e[b - 1] * V[b - 1] if b else 0.0)
            if b:
                total += 1
                lam, z = np.linalg.eigh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
                x = np.array(V).T @ z[:, 0]
                if abs(E - lam[0]) < ACC:
                    return total, lam[0], x / np.linalg.norm(x), lam[1] - lam[0]
                if b < block - 1:   # (a restart does not update the energy)
                    E = lam[0]
            e.append(np.linalg.norm(w))
            V.append(w / e[b])
        w = x


@pytest.mark.parametrize("block", [800, 12])
@pytest.mark.parametrize("which", [40, 257, 2100, "superblock"])
def test_lanczos_recurrence(gpu, which, block):
    A = _superblock() if which == "superblock" else _random(which)
    A.sort_indices()
    n, norm = A.shape[0], abs(A).sum(axis=1).max()
    guess = np.random.default_rng(1).standard_normal(n)
    steps, energy, x, gap = _lanczos(A, guess.copy(), block)
    assert steps <= 80
    p = gpu.default_params(dense_below=0, lanczos_acc=ACC, lanczos_block_step=block)
    m = gpu.DeviceMatrix(abi.Crs.from_scipy(A))
    for shape in (None, 1, 2, 4, 8, "csr"):
        if shape == "csr":
            m.set_format(gpu.DG_FORMAT_CSR)
        elif shape:
            m.set_sell_shape(shape, 3 if n < 1000 else 150)
        v, info = gpu.ground_state(m, p, guess=guess, lanczos_only=True)
        assert info.converged and info.dense == 0 and info.lanczos_steps == steps, shape
        assert abs(info.eig_val - energy) <= 1e-12 * norm, shape
        assert np.linalg.norm(v - np.copysign(1.0, v @ x) * x) <= 1e-12 * norm / gap, shape
