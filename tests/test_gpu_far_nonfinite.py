"""NaN and infinite densities in the several-density products (GPU): one such
value at one node makes every potential of its own density NaN or infinite and
leaves the other densities as they are, whichever kernels take the far field."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0, 1], ids=["lap", "helm"])
def plan(request):
    from fmm3dbie_b200 import Plan
    kind = request.param
    s = S.torus_quad(7, 5, 4)
    zp = (2.0, -2.0j, 1.0) if kind else (1.0, 1.0)
    st = S.setup(s, kind, 1e-7, zp)
    P = Plan(kind, zp, s, st.near, st.over)
    yield P, kind, s.npts
    P.close()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nd", [2, 5, 16, 33, 64])
def test_bad_value_is_kept(plan, nd, prec, bad):
    import torch
    P, kind, n = plan
    g = torch.Generator(device="cpu").manual_seed(nd)
    x = torch.randn(n, nd, generator=g, dtype=torch.complex128 if kind else torch.float64).cuda()
    m = nd // 2
    y = x.clone()
    y[n // 3, m] = bad
    rest = [q for q in range(nd) if q != m]
    for variant in (0, 1, 2, 3, 4):
        P.set_far(prec, nd, variant, 2)
        clean, got = P.matvec(x, prec), P.matvec(y, prec)
        assert bool((~torch.isfinite(got[:, m])).all()), variant
        assert torch.equal(got[:, rest], clean[:, rest]), variant
