"""A solve that gives up while its kernels are still queued, beside solves on other threads: what it
leaves behind (its pinned blocks, and with its thread its stream) must not reach them before its last
kernel has run.  Runs in a process of its own with a short bound on the waits (20 ms); the solve that gives
up has a product of one block (62 ms), and the others wait some tens of microseconds.  All kernels are
loaded beforehand (loading one waits for the kernels that run) and every stream has a work queue of its
own."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

SCRIPT = """
import sys, threading, time
import numpy as np
from dmrg_c_gb300 import lib as gpu
from dmrg_c_gb300.ed_models import xxz_chain

ends = sys.argv[1] == "ends"      # the thread that gives up ends (its stream is handed on) or stays
small = [gpu.EDSystem(xxz_chain(14, Jz=0.3 + 0.2 * k)).matrix() for k in range(6)]
p = gpu.default_params(seed=5)
want = [gpu.ground_state(m, p) for m in small]
big = gpu.EDSystem(xxz_chain(24, Jz=0.5)).matrix()
big.set_sell_shape(1, 1)
out = np.empty(big.n)
gave_up, done = threading.Event(), threading.Event()
failure = []

def abandoned():
    try:
        gpu.ground_state(big, gpu.default_params(seed=1, lookahead=8), out=out)
    except gpu.DgError as e:
        failure.append(str(e))
    gave_up.set()
    if not ends:
        done.wait()

t = threading.Thread(target=abandoned, daemon=True)
t.start()
gave_up.wait()
if ends:
    t.join()
t0 = time.perf_counter()
for _ in range(24):
    got = [None] * len(small)

    def solve(k):
        got[k] = gpu.ground_state(small[k], p)

    threads = [threading.Thread(target=solve, args=(k,)) for k in range(len(small))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for (v, info), (w, ref) in zip(got, want):
        assert info.eig_val == ref.eig_val and info.lanczos_steps == ref.lanczos_steps
        assert np.array_equal(v, w)
assert time.perf_counter() - t0 < 0.5   # well before the abandoned steps end
time.sleep(3.0)                   # the abandoned kernels still read the matrix
done.set()
t.join()
assert failure and "timed out" in failure[0], failure
print("ok")
"""


@pytest.mark.parametrize("thread", ["stays", "ends"])
def test_abandoned_solve(gpu, thread):
    env = dict(os.environ, DG_WAIT_TIMEOUT_MS="20", CUDA_MODULE_LOADING="EAGER", CUDA_DEVICE_MAX_CONNECTIONS="32",
               PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", SCRIPT, thread], cwd=ROOT, env=env, capture_output=True, text=True, timeout=120)
    print(r.stdout)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
