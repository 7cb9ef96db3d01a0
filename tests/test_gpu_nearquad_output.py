"""Where the near quadrature's result may go (GPU): pageable and pinned host
arrays, and device memory, which the host must not touch while the kernel
runs (the copy at the end is the runtime's to do or to refuse)."""
import ctypes as C

import numpy as np
import pytest

from fmm3dbie_b200 import _lib as L
from fmm3dbie_b200 import surface as S

pytestmark = pytest.mark.gpu


def _call(s, st, params, wnear):
    n = st.near
    ids, uvs = s.patch_id_uvs()
    ids, uvs = np.ascontiguousarray(ids, np.int64), np.ascontiguousarray(uvs, float)
    rad = np.zeros(4, np.int64)
    targs = np.ascontiguousarray(s.srcvals, float)
    return L.lib().bie_getnearquad_lap_comb_dir_eval_gpu(
        s.npatches, L.ptr(s.norders), L.ptr(s.ixyzs), L.ptr(s.iptype), s.npts, L.ptr(s.srccoefs),
        L.ptr(s.srcvals), targs.shape[1], s.npts, L.ptr(targs), L.ptr(ids), L.ptr(uvs), 1e-6,
        L.ptr(params), 1, n.col_ind.shape[0], L.ptr(n.row_ptr), L.ptr(n.col_ind), L.ptr(n.iquad),
        0.0, n.wnear.size, C.cast(wnear, L.PDBL), L.ptr(rad))


@pytest.mark.parametrize("where", ["pageable", "pinned", "device"])
def test_output_memory(where):
    import torch
    s = S.torus_quad(14, 8, 5)
    params = np.array([1.0, 1.0])
    st = S.setup(s, 0, 1e-6, params)
    n = st.near.wnear.size
    assert 8 * n > 2 * (4 << 20)  # large enough for the staged copy
    out = torch.zeros(n, dtype=torch.float64, device="cuda" if where == "device" else "cpu",
                      pin_memory=where == "pinned")
    status = _call(s, st, params, out.data_ptr())
    if where != "device":
        assert status == 0
    if status == 0:
        ref = st.near.wnear
        assert np.linalg.norm(out.cpu().numpy() - ref) <= 1e-13 * np.linalg.norm(ref)
    else:
        assert status == 2
    print(f"\n{where}: status {status}")
