"""FP32 Laplace products of 2 to 8 densities in the shape for few targets (GPU):
target counts around its 128-target blocks, density counts that fill a block's
group and that do not.  Reference: the paired shape with the same chunks, whose
pairs and tile sums are the same operations in the same order, and the FP64
product within the paired shape's own error."""
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 1), (4, 4, 2), (8, 4, 1), (7, 3, 2), (14, 8, 4)])
@pytest.mark.parametrize("nd", [2, 3, 4, 5, 7, 8])
def test_small_shape(monkeypatch, shape, nd):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(*shape)
    zp = (1.0, 0.5)
    st = S.setup(s, 0, 1e-6, zp)
    g = torch.Generator(device="cpu").manual_seed(nd)
    x = torch.randn(s.npts, nd, generator=g, dtype=torch.float64).cuda()
    P = Plan(0, zp, s, st.near, st.over)
    y64 = P.matvec(x, 0)
    monkeypatch.setenv("BIE_FAR_VARIANT", "5")
    small = P.matvec(x, 1)
    variant, nchunks, _ = P.get_far(1, nd)
    assert variant == 5
    P.set_far(1, nd, 0, nchunks)
    pairs = P.matvec(x, 1)
    P.close()

    def rel(a, b):
        return float(((a - b).norm(dim=0) / b.norm(dim=0)).max())

    assert rel(small, pairs) < 2.0 ** -22
    assert rel(small, y64) < 1.05 * rel(pairs, y64) + 2.0 ** -24
