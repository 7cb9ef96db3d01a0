"""Direct far field of small problems (GPU): the 32-target shape (targets that
leave a partial block, chunks that leave a partial tile, targets past the first
512-target block whose FP32 coordinates are centred on their own) against the
other shapes."""
import numpy as np
import pytest

from fmm3dbie_b200 import BieError
from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu

# FP64: the same pair function, summed in another order.  FP32: the same pair
# values, tile sums of 32 instead of 128 sources in two lanes: rounding of the
# FP32 tile sums only.
TOL = {0: 1e-13, 1: 2e-6}


@pytest.mark.parametrize("kind,params", [(0, (1.0, 0.5)), (1, (2.0, -2.0j, 1.0)),
                                         (1, (1.0 + 0.5j, -1.0j, 1.0))])
@pytest.mark.parametrize("shape", [(3, 2, 2), (5, 3, 4), (9, 5, 4), (13, 6, 5)])
def test_small_shape(kind, params, shape, monkeypatch):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(*shape)
    st = S.setup(s, kind, 1e-6, params)
    g = torch.Generator(device="cpu").manual_seed(1)
    dt = torch.float64 if kind == 0 else torch.complex128
    x = torch.randn(s.npts, generator=g, dtype=dt).cuda()
    ref = {}
    P = Plan(kind, params, s, st.near, st.over)
    most = (P.nptso + 127) // 128
    for prec in (0, 1):
        P.set_far(prec, 1, 0, 1)
        ref[prec] = P.matvec(x, prec)
    with pytest.raises(BieError):
        P.set_far(0, 1, 5, 1)
    P.close()
    monkeypatch.setenv("BIE_FAR_VARIANT", "5")
    monkeypatch.setenv("BIE_AUTOTUNE", "0")
    for waves in ("0.01", "1", "1000"):
        monkeypatch.setenv("BIE_FAR_WAVES", waves)
        P = Plan(kind, params, s, st.near, st.over)
        for prec in (0, 1):
            assert P.get_far(prec, 1)[0] == 5 and P.get_far(prec, 1)[1] <= most
            y = P.matvec(x, prec)
            assert float((y - ref[prec]).norm()) < TOL[prec] * float(ref[prec].norm())
        P.close()
