"""Orthogonalisation of several systems (GPU) at the edge between the reduction
in the last block and the one over the chip: 32 outputs (vectors times
systems), reached with one vector or within a solve.  Reference: each system
solved on its own; both stop at residuals below eps, so the solutions differ
by at most 2 eps times the condition number (< 100)."""
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu
EPS = 1e-10


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("nd", [2, 8, 31, 32, 33, 40, 200])
def test_systems(kind, nd):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(6, 4, 4)
    zp = (1.0, -1.0j, 1.0) if kind else (1.0, 0.0)
    st = S.setup(s, kind, 1e-4, zp)
    P = Plan(kind, zp, s, st.near, st.over)
    g = torch.Generator(device="cpu").manual_seed(nd)
    b = torch.randn(s.npts, nd, generator=g, dtype=torch.complex128 if kind else torch.float64).cuda()
    x, info = P.solve(b, 0.5, numit=150, eps_gmres=EPS)
    assert info["status"] == 0
    for q in sorted({0, 1, nd // 2, nd - 1}):
        one, i1 = P.solve(b[:, q].contiguous(), 0.5, numit=150, eps_gmres=EPS)
        assert abs(int(i1["niter"][0]) - int(info["niter"][q])) <= 1
        assert float((one - x[:, q]).norm()) < 200 * EPS * float(one.norm())
    P.close()
