"""Memory of the several-density FP32 products (GPU): the tensor-core far
field's density operand is held only by plans that use one of its shapes."""
import numpy as np
import pytest

from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


def test_operand_only_where_it_is_read():
    import torch
    from fmm3dbie_b200 import Plan
    s = S.torus_quad(28, 16, 5)
    zp = (2.0, -2.0j, 1.0)
    st = S.setup(s, 1, 1e-5, zp)
    nd = 64
    x = torch.ones(s.npts, nd, dtype=torch.complex128, device="cuda")
    out = torch.empty_like(x)
    used = {}
    for variant in (0, 4):
        P = Plan(1, zp, s, st.near, st.over)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        P.set_far(1, nd, variant, 1)
        P.matvec(x, 1, out=out)
        torch.cuda.synchronize()
        used[variant] = before - torch.cuda.mem_get_info()[0]
        operand = (P.nptso + 63) // 64 * 64 * nd * 4 * 4  # (re, im) x (high, low) in FP32
        P.close()
    print(f"\nCUDA cores {used[0] / 2**20:.0f} MB, tensor cores {used[4] / 2**20:.0f} MB, "
          f"operand {operand / 2**20:.0f} MB")
    assert used[4] - used[0] >= operand
