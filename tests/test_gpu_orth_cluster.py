"""Orthogonalisation of one small system by a cluster (GPU): slices of unequal
length, more and fewer vectors than warps, more vectors than one launch of it
takes, systems that grow past its range.  Reference: the same system solved
as one of two (the chip-wide kernels).  Both stop at residuals below eps, so
the solutions differ by at most 2 eps times the condition number (< 100)."""
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu
EPS = 1e-10


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("shape,zid", [((3, 3, 1), 0.5), ((6, 4, 4), 0.5), ((7, 5, 6), 0.05),
                                       ((9, 5, 4), 0.02), ((28, 16, 5), 0.5)])
def test_single_system(kind, shape, zid):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(*shape)
    zp = (1.0, -1.0j, 1.0) if kind else (1.0, 0.0)
    st = S.setup(s, kind, 1e-4, zp)
    P = Plan(kind, zp, s, st.near, st.over)
    g = torch.Generator(device="cpu").manual_seed(s.npts)
    b = torch.randn(s.npts, 2, generator=g, dtype=torch.complex128 if kind else torch.float64).cuda()
    two, i2 = P.solve(b, zid, numit=150, eps_gmres=EPS)
    one, i1 = P.solve(b[:, 0].contiguous(), zid, numit=150, eps_gmres=EPS)
    n1, n2 = int(i1["niter"][0]), int(i2["niter"][0])
    assert abs(n1 - n2) <= 1
    assert float((one - two[:, 0]).norm()) < 200 * EPS * float(two[:, 0].norm())
    P.close()


def test_zero_right_hand_side():
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(6, 4, 4)
    st = S.setup(s, 0, 1e-4, (1.0, 0.0))
    P = Plan(0, (1.0, 0.0), s, st.near, st.over)
    x, info = P.solve(torch.zeros(s.npts, dtype=torch.float64, device="cuda"), 0.5)
    assert float(x.abs().max()) == 0.0 and int(info["niter"][0]) == 0
    P.close()
