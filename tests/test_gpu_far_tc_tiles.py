"""Tensor-core far field at the edges of its tiles and density groups (GPU):
density counts around the 16/32/64-column groups, source counts that leave a
partial 64-source tile in the last chunk, target counts that leave a partial
128-target block, one chunk to one chunk per 128 sources, a complex
wavenumber.  Reference: the FP64 matvec and the CUDA-core FP32 kernels."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu

# An accumulator takes at most 8 hi*hi steps, each losing less than one unit
# in the last place (2^-23) of the accumulator; the rest of the error is the
# FP32 pair arithmetic that both kernels share.
STEPS = 8 * 2.0 ** -23


@pytest.mark.parametrize("zk", [2.0, 1.5 + 0.5j])
@pytest.mark.parametrize("shape", [(4, 3, 3), (5, 4, 4), (7, 5, 2)])
def test_tile_edges(shape, zk):
    import torch
    from fmm3dbie_b200 import Plan
    nu, nv, norder = shape
    s = S.torus_quad(nu, nv, norder)
    zp = (zk, -1j * zk, 1.0)
    st = S.setup(s, 1, 1e-7, zp)
    P = Plan(1, zp, s, st.near, st.over)
    w = torch.tensor(s.qwts(), device="cuda")[:, None]

    def rel(a, b):
        return float(((w * (a - b).abs() ** 2).sum(0) / (w * b.abs() ** 2).sum(0)).sqrt().max())

    most = (P.nptso + 127) // 128
    for nd in (2, 3, 15, 16, 17, 32, 33, 64, 65):
        g = torch.Generator(device="cpu").manual_seed(nd)
        x = torch.randn(s.npts, nd, generator=g, dtype=torch.complex128).cuda()
        y64 = P.matvec(x, 0)
        P.set_far(1, nd, 0, 1)
        e_simt = rel(P.matvec(x, 1), y64)
        for variant in (3, 4):
            for nchunks in sorted({1, min(3, most), most}):
                P.set_far(1, nd, variant, nchunks)
                y = P.matvec(x, 1)
                torch.cuda.synchronize()
                assert P.get_far(1, nd)[2] == 0, "completion wait timed out"
                assert rel(y, y64) < 1.5 * e_simt + STEPS, (nd, variant, nchunks, e_simt)
    P.close()
