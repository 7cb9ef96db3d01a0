"""Setups and plan builds in several threads at once (GPU): results on their
way to the host and the arrays of a plan build are staged apart, and a thread
that finds a staging buffer in use gets the same values without it."""
import threading

import numpy as np
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


def test_threads():
    import torch
    from fmm3dbie_b200 import Plan
    zp = (2.0, -2.0j, 1.0)
    s = S.torus_quad(14, 8, 6)
    st = S.setup(s, 1, 1e-7, zp)
    assert st.near.wnear.nbytes > 2 * (4 << 20)  # large enough for the staged copy
    x = torch.ones(s.npts, dtype=torch.complex128, device="cuda")
    P = Plan(1, zp, s, st.near, st.over)
    ref = P.matvec(x, 0).cpu().numpy()
    P.close()
    errs = []
    barrier = threading.Barrier(5)

    def check(got, want):
        d = np.linalg.norm(got - want) / np.linalg.norm(want)
        if not d < 1e-13:
            errs.append(d)

    def setups():
        try:
            barrier.wait()
            for _ in range(3):
                check(S.setup(s, 1, 1e-7, zp).near.wnear, st.near.wnear)
        except Exception as e:  # reported below, in the test's own thread
            errs.append(e)

    def builds():
        try:
            barrier.wait()
            for _ in range(3):
                Q = Plan(1, zp, s, st.near, st.over)
                check(Q.matvec(x, 0).cpu().numpy(), ref)
                Q.close()
        except Exception as e:
            errs.append(e)

    th = [threading.Thread(target=f) for f in (setups, setups, setups, builds, builds)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errs, errs
