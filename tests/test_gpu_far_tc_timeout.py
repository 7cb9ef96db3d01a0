"""A wait of the tensor-core far field that runs out (GPU): the launch ends, its
potentials are NaN instead of what the buffer held before, a solve reports a
breakdown, and the plan goes on as if nothing had been once waits may take
their time again.  The waits are made to run out by a limit of no polls; no
fault is involved."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd,variant", [(4, 3), (20, 3), (64, 4)])
def test_wait_runs_out(nd, variant):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(8, 5, 4)
    zp = (2.0, -2.0j, 1.0)
    st = S.setup(s, 1, 1e-7, zp)
    P = Plan(1, zp, s, st.near, st.over)
    g = torch.Generator(device="cpu").manual_seed(nd)
    x = torch.randn(s.npts, nd, generator=g, dtype=torch.complex128).cuda()
    P.set_far(1, nd, variant, 3)
    good = P.matvec(x, 1).clone()
    assert P.get_far(1, nd)[2] == 0
    P.set_tc_wait(0)
    bad = P.matvec(x, 1)
    torch.cuda.synchronize()
    assert bool(torch.isnan(bad.real).all()) and P.get_far(1, nd)[2] != 0
    _, info = P.solve(x, 0.5, mode=1, eps_gmres=1e-8)
    assert info["status"] == 4
    P.set_tc_wait()
    assert torch.equal(P.matvec(x, 1), good)
    _, info = P.solve(x, 0.5, mode=1, eps_gmres=1e-8)
    assert info["status"] == 0 and float(np.max(info["rres"])) < 1e-8
    P.close()
