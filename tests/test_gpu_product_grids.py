"""The grid of the FP32 (mixed) product is its own: tuning the shapes, or setting a variant or the warps
per slice, leaves it at the default of its warps per slice, whatever the FP64 product's grid becomes.  The
grid groups the sums of the mixed Lanczos, so a tuned matrix and a fresh one with the same FP32 shape give
the same bits."""
import numpy as np
import pytest
import scipy.sparse as sp

from dmrg_c_gb300 import abi

pytestmark = pytest.mark.gpu

V_U16, V_PIPE8 = 2, 3


def _banded(n, bands, seed):
    """Symmetric, 2 * bands + 1 elements a row, one low state."""
    rng = np.random.default_rng(seed)
    off = np.sort(rng.choice(np.arange(1, 5000), bands, replace=False))
    r, c, v = [np.arange(n)], [np.arange(n)], [rng.uniform(0, 1, n)]
    for d in off:
        x = 0.2 * rng.uniform(-1, 1, n - d)
        r += [np.arange(n - d), np.arange(d, n)]
        c += [np.arange(d, n), np.arange(n - d)]
        v += [x, x]
    v[0][n // 3] = -9.0
    A = sp.csr_matrix((np.concatenate(v), (np.concatenate(r), np.concatenate(c))), shape=(n, n))
    A.sort_indices()
    return abi.Crs.from_scipy(A)


@pytest.fixture(scope="module")
def operator():
    return _banded(150_016, 16, 3)   # more slices than three blocks a SM take


def _fresh(gpu, operator):
    return gpu.DeviceMatrix(operator, gpu.DG_STORE_FULL, gpu.DG_VALUES_BOTH)


def _mixed(gpu, m, mixed):
    v, info = gpu.ground_state(m, gpu.default_params(seed=4, mixed=mixed, lanczos_max_step=40, lanczos_block_step=40, lanczos_acc=1e-6),
                               lanczos_only=True)
    return info.eig_lanczos, info.lanczos_steps, v


def _same(a, b):
    assert a[0] == b[0] and a[1] == b[1] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("mixed", [1, 2])
def test_tuning_keeps_the_fp32_grid(gpu, operator, mixed):
    gpu.shape_cache_clear()
    tuned = _fresh(gpu, operator)
    assert tuned.shape_cache_apply(tune=True, iters=2) == 2
    c = tuned.sell_config()
    plain = _fresh(gpu, operator)
    plain.set_sell_mixed(c["ws32"], c["variant32"])
    _same(_mixed(gpu, tuned, mixed), _mixed(gpu, plain, mixed))
    other = _fresh(gpu, operator)   # the class applied, not tuned
    assert other.shape_cache_apply(tune=False) == 1
    _same(_mixed(gpu, tuned, mixed), _mixed(gpu, other, mixed))
    gpu.shape_cache_clear()


def test_variant_takes_its_own_grid(gpu, operator):
    """The pipelined FP64 form runs three blocks a SM, the others as many as the slices need (up to
    sixteen a SM); a grid that the caller gave stays."""
    m = _fresh(gpu, operator)

    def config():
        c = m.sell_config()
        return c["ws"], c["grid"], c["variant"]

    ws, grid, variant = config()
    need = -(-4736 // (8 // ws))   # (slices of 32 rows, whole windows of 2,048 rows)
    assert variant == V_PIPE8 and grid < need
    m.set_sell_variant(V_U16)
    assert config() == (ws, need, V_U16)
    m.set_sell_window(32)
    assert config() == (ws, need, V_U16)
    m.set_sell_variant(V_PIPE8)
    assert config() == (ws, grid, V_PIPE8)
    m.set_sell_shape(2, 77)
    m.set_sell_variant(V_U16)
    assert config() == (2, 77, V_U16)
