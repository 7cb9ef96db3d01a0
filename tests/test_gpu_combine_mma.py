"""Near correction of many complex densities by matrix instructions (GPU):
rows that leave a partial group of 8, densities that leave a partial group of
16, patches whose node count is no multiple of 4, near lists in ascending and
in descending order.  Reference: the same densities 7 at a time (another form of
the near correction)."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S
from fmm3dbie_b200.surface import NearField

pytestmark = pytest.mark.gpu


def reversed_rows(near):
    """The same near quadrature with every row's pairs in reverse order."""
    n = np.diff(near.iquad)
    order = np.concatenate([np.arange(b - 2, a - 2, -1)
                            for a, b in zip(near.row_ptr[:-1], near.row_ptr[1:])]).astype(np.int64)
    w = np.concatenate([near.wnear[near.iquad[q] - 1:near.iquad[q] - 1 + n[q]] for q in order])
    iquad = np.concatenate([[1], 1 + np.cumsum(n[order])]).astype(np.int64)
    return NearField(near.row_ptr, np.ascontiguousarray(near.col_ind[order]), iquad, w)


@pytest.mark.parametrize("shape,nd", [((9, 5, 4), 200), ((12, 7, 4), 97), ((13, 6, 5), 120)])
@pytest.mark.parametrize("descending", [False, True])
def test_many_densities(shape, nd, descending):
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(*shape)
    zp = (2.0, -2.0j, 1.0)
    st = S.setup(s, 1, 1e-6, zp)
    assert (s.npts + 7) // 8 * ((nd + 15) // 16) >= 1536  # the form under test
    near = reversed_rows(st.near) if descending else st.near
    P = Plan(1, zp, s, near, st.over)
    Q = Plan(1, zp, s, st.near, st.over)
    g = torch.Generator(device="cpu").manual_seed(nd)
    x = torch.randn(s.npts, nd, generator=g, dtype=torch.complex128).cuda()
    for prec, tol in ((0, 1e-12), (1, 2e-6)):  # FP32: two forms of the FP32 far field
        y = P.matvec(x, prec)
        ref = torch.cat([Q.matvec(x[:, m:m + 7].contiguous(), prec) for m in range(0, nd, 7)], 1)
        assert float((y - ref).norm()) < tol * float(ref.norm()), prec
    P.close()
    Q.close()
