"""dg_release_pool hands back the pinned host blocks that solves leave in the library's list (they show in the
process' mapped memory), also those of threads that have ended, and solves after it are the same."""
import threading

import numpy as np
import pytest

from dmrg_c_gb300.ed_models import xxz_chain

pytestmark = pytest.mark.gpu


def _mapped_bytes():
    with open("/proc/self/status") as f:
        return next(1024 * int(line.split()[1]) for line in f if line.startswith("VmSize"))


def test_pinned_blocks_go_back(gpu):
    m = gpu.EDSystem(xxz_chain(12, Jz=0.4)).matrix()
    plain = gpu.default_params(seed=3, dense_below=0)
    want, ref = gpu.ground_state(m, plain)
    # mirrors for 2^20 + 1 steps: three blocks of 16 MiB
    p = gpu.default_params(seed=3, dense_below=0, lanczos_max_step=1 << 20, lanczos_block_step=1 << 20)
    t = threading.Thread(target=gpu.ground_state, args=(m, p))
    t.start()
    t.join()
    before = _mapped_bytes()
    assert gpu.load().dg_release_pool() == 0
    assert before - _mapped_bytes() >= 32 << 20
    v, info = gpu.ground_state(m, plain)
    assert info.eig_val == ref.eig_val and np.array_equal(v, want)
