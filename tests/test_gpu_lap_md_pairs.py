"""FP32 Laplace far field of several densities (GPU), two targets per packed
instruction: density counts around its groups of 4 and 8, target counts that
leave partial blocks, source counts that leave partial tiles, in a plan and in
a batch of uneven surfaces.  Reference: FP64 (FP32 pair arithmetic and tile
sums of 128 sources: a few 1e-7)."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S
from fmm3dbie_b200.batch import BatchItem, SurfaceBatch

pytestmark = pytest.mark.gpu

SHAPES = [(3, 2, 2), (6, 4, 3), (11, 5, 4)]


@pytest.mark.parametrize("shape", SHAPES)
def test_plan(shape):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(*shape)
    st = S.setup(s, 0, 1e-6, (1.0, 0.7))
    P = Plan(0, (1.0, 0.7), s, st.near, st.over)
    most = (P.nptso + 127) // 128
    for nd in (2, 3, 4, 5, 8, 9, 17):
        g = torch.Generator(device="cpu").manual_seed(nd)
        x = torch.randn(s.npts, nd, generator=g, dtype=torch.float64).cuda()
        ref = P.matvec(x, 0)
        for variant in (0, 1, 2):
            for nchunks in sorted({1, most}):
                P.set_far(1, nd, variant, nchunks)
                err = float((P.matvec(x, 1) - ref).norm() / ref.norm())
                assert err < 2e-6, (nd, variant, nchunks, err)
    P.close()


@pytest.mark.parametrize("nd", [1, 3, 4, 8, 12])
def test_batch(nd):
    import torch
    items = [BatchItem(S.torus_quad(*sh), 0, (1.0, 0.7), 0.5) for sh in SHAPES]
    B = SurfaceBatch(items, 1e-6)
    n = sum(it.surf.npts for it in items)
    g = torch.Generator(device="cpu").manual_seed(nd)
    x = torch.randn(n, nd, generator=g, dtype=torch.float64).cuda()
    ref, y = B.matvec(x, 0), B.matvec(x, 1)
    for a, b in zip(B.split(y), B.split(ref)):
        assert float((a - b).norm()) < 2e-6 * float(b.norm())
    B.close()
