"""Tensor-core far field over long source chunks (GPU): the error of a sum does
not grow with the number of tiles it runs over.  Reference: the FP64 matvec.

One chunk of all sources is compared with chunks of 8 tiles, whose sums go to
FP64.  Every 8 tiles a running sum is folded away without loss, so the two
differ by the FP32 additions within 8 tiles: each rounds by at most 2^-24 of a
sum over a small part of the sources, with either sign."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd,variant", [(64, 4), (48, 4), (32, 3), (16, 3)])
def test_long_chunk(nd, variant):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(28, 16, 5)
    zk = 2.0
    zp = (zk, -1j * zk, 1.0)
    st = S.setup(s, 1, 1e-7, zp)
    P = Plan(1, zp, s, st.near, st.over)
    w = torch.tensor(s.qwts(), device="cuda")[:, None]
    d = np.random.default_rng(nd).normal(size=(nd, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    x = torch.tensor(np.exp(1j * zk * (s.srcvals[:, :3] @ d.T)), device="cuda")
    y64 = P.matvec(x, 0)

    def err(nchunks):
        P.set_far(1, nd, variant, nchunks)
        y = P.matvec(x, 1)
        return float(((w * (y - y64).abs() ** 2).sum(0) / (w * y64.abs() ** 2).sum(0)).sqrt().max())

    short, long = err(max(1, P.nptso // 512)), err(1)
    print(f"\n{nd} densities: chunks of 8 tiles {short:.2e}, one chunk {long:.2e}")
    assert long <= short + 2.0 ** -24
    P.close()
