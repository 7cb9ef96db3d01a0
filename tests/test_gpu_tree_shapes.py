"""Hierarchical far field over the shapes its kernels split by (GPU): target
leaves of one to four warps (one to six parts of a source tile), source leaves
that leave partial tiles, grids of 1 to 16 points a side (every compiled count
of the upward pass), real and complex wavenumbers.  Reference: the direct
matvec."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


def bound(p, prec):
    """Chebyshev interpolation of a source at r / theta = 2 r from a box of
    half diagonal r: ratio 2 + sqrt(3) per point; FP32 adds its rounding."""
    return 10.0 * (2.0 + 3.0 ** 0.5) ** -(p - 1) + (2e-6 if prec else 1e-11)


@pytest.fixture(scope="module", params=[(0, (1.0, 1.0)), (1, (2.0, -2.0j, 1.0)),
                                        (1, (1.0 + 0.3j, -1.0j, 1.0))],
                ids=["lap", "helm", "helm_ck"])
def plan(request):
    import torch
    from fmm3dbie_b200 import Plan
    kind, params = request.param
    s = S.torus_quad(14, 7, 4)
    st = S.setup(s, kind, 1e-7, params)
    P = Plan(kind, params, s, st.near, st.over)
    x = np.random.default_rng(0).normal(size=s.npts)
    x = torch.tensor(x if kind == 0 else x * np.exp(1j * np.arange(s.npts)), device="cuda")
    ref = P.matvec(x, 0)
    yield P, x, ref
    P.close()


@pytest.mark.parametrize("leaf_t,leaf_s,p", [(1, 4, 3), (16, 32, 5), (33, 50, 6), (64, 64, 7),
                                             (70, 130, 8), (96, 200, 10), (128, 256, 12),
                                             (128, 500, 16), (40, 300, 14), (128, 20, 9)])
def test_tree_shapes(plan, leaf_t, leaf_s, p):
    P, x, ref = plan
    for prec in (0, 1):
        P.set_far_method(prec, 1, 0.5, p, leaf_t, leaf_s)
        err = float((P.matvec(x, prec) - ref).norm() / ref.norm())
        P.set_far_method(prec, 0)
        assert err < bound(p, prec), (prec, err)


def test_trig_table_phases():
    """FP64 phases over the table's octants and past one turn: a single-layer
    matvec with growing wavenumber against the oracle's direct sum."""
    import oracle
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(6, 4, 3)
    for zk in (0.01, 1.0, 7.0, 17.0):
        zp = (zk, 1.0, 0.5)
        st = S.setup(s, 1, 1e-5, zp)
        sig = np.random.default_rng(1).normal(size=s.npts) * (1.0 + 0.5j)
        P = Plan(1, zp, s, st.near, st.over)
        got = P.matvec(torch.tensor(sig, device="cuda"), 0).cpu().numpy()
        ref = oracle.lpcomp(1, s, zp, st.near, st.over, sig)
        P.close()
        assert np.linalg.norm(got - ref) < 1e-12 * np.linalg.norm(ref), zk
