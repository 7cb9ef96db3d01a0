"""Near correction of many complex densities with vectors at an 8-byte boundary
(GPU): the matrix-instruction form moves 16 bytes at a time, so such calls take
the form that does not.  Reference: the same product of aligned vectors."""
import pytest

from fmm3dbie_b200 import _lib as L
from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plan():
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(14, 8, 6)
    zp = (2.0, -2.0j, 1.0)
    st = S.setup(s, 1, 1e-6, zp)
    P = Plan(1, zp, s, st.near, st.over)
    yield P
    P.close()


@pytest.mark.parametrize("shift_in,shift_out", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nd", [40, 64])
def test_eight_byte_boundary(plan, nd, prec, shift_in, shift_out):
    import torch
    P = plan
    assert (P.npts + 7) // 8 * ((nd + 15) // 16) >= 1536  # the matrix form's range
    g = torch.Generator(device="cpu").manual_seed(nd)
    x = torch.randn(P.npts, nd, generator=g, dtype=torch.complex128).cuda()
    want = torch.view_as_real(P.matvec(x, prec)).reshape(-1)
    n = want.numel()
    src = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    dst = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    src[shift_in:shift_in + n] = torch.view_as_real(x).reshape(-1)
    stream = torch.cuda.current_stream().cuda_stream
    L.check(L.lib().bie_plan_matvec(P._h, prec, nd, src.data_ptr() + 8 * shift_in,
                                    dst.data_ptr() + 8 * shift_out, stream), "bie_plan_matvec")
    got = dst[shift_out:shift_out + n]
    assert float((got - want).norm() / want.norm()) < 1e-13
