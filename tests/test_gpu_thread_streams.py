"""Streams and pinned blocks handed from threads that ended to later ones: solves from many
short-lived threads, one after another and at the same time, give what one thread gives."""
import threading

import numpy as np
import pytest

from dmrg_c_gb300.ed_models import xxz_chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at_once", [1, 8])
def test_solves_from_short_lived_threads(gpu, at_once):
    mats = [gpu.EDSystem(xxz_chain(14, Jz=0.3 + 0.2 * k)).matrix() for k in range(at_once)]
    p = gpu.default_params(seed=5)
    want = [gpu.ground_state(m, p) for m in mats]
    for _ in range(96 // at_once):
        got = [None] * at_once

        def solve(k):
            got[k] = gpu.ground_state(mats[k], p)

        threads = [threading.Thread(target=solve, args=(k,)) for k in range(at_once)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for (v, info), (w, ref) in zip(got, want):
            assert info.eig_val == ref.eig_val
            assert np.array_equal(v, w)
