"""FP64 far field of many densities by matrix instructions (GPU): density counts
around its groups of 16, 32 and 64 columns, target counts that leave partial
64-target blocks, source counts that leave partial 32-source tiles, one chunk
to one per 128 sources, a complex wavenumber.  Reference: the CUDA-core kernel
(the same pair values, summed in another order)."""
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zk", [2.0, 1.5 + 0.5j])
@pytest.mark.parametrize("shape", [(3, 2, 2), (5, 4, 3), (9, 4, 5)])
def test_matches_cuda_cores(shape, zk):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(*shape)
    zp = (zk, -1j * zk, 1.0)
    st = S.setup(s, 1, 1e-6, zp)
    P = Plan(1, zp, s, st.near, st.over)
    most = (P.nptso + 127) // 128
    for nd in (9, 15, 16, 17, 32, 33, 63, 64, 65, 100):
        g = torch.Generator(device="cpu").manual_seed(nd)
        x = torch.randn(s.npts, nd, generator=g, dtype=torch.complex128).cuda()
        P.set_far(0, nd, 0, 1)
        ref = P.matvec(x, 0)
        for variant in (3, 4):
            for nchunks in sorted({1, min(3, most), most}):
                P.set_far(0, nd, variant, nchunks)
                y = P.matvec(x, 0)
                # FP64 sums of a few thousand terms in another order
                assert float((y - ref).norm()) < 1e-12 * float(ref.norm()), (nd, variant, nchunks)
    P.close()
