"""Host side of a single system's solve (GPU): a process that asked CUDA for
blocking waits gets them, its thread does not spin through the products."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SRC = """
import ctypes, time
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
assert cu.cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0  # CU_CTX_SCHED_BLOCKING_SYNC
import numpy as np, torch
from fmm3dbie_b200 import Plan, surface as S
s = S.torus_quad(28, 16, 5)
zp = (2.0, -2.0j, 1.0)
st = S.setup(s, 1, 1e-5, zp)
P = Plan(1, zp, s, st.near, st.over)
b = torch.tensor(np.exp(1j * s.srcvals[:, 0]), device="cuda")
P.solve(b, 0.5, eps_gmres=1e-8)
torch.cuda.synchronize()
w, c = time.perf_counter(), time.thread_time()
x, info = P.solve(b, 0.5, eps_gmres=1e-8)
w, c = time.perf_counter() - w, time.thread_time() - c
print("times", w, c, int(info["niter"][0]))
"""


def test_blocking_waits():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SRC], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    wall, cpu, niter = (float(v) for v in r.stdout.split("times")[1].split())
    print(f"\n{niter:.0f} iterations, {1e3 * wall:.1f} ms, {1e3 * cpu:.1f} ms of the thread")
    # an iteration's launches take the thread some 30 us of more than a millisecond
    assert cpu < 0.5 * wall
