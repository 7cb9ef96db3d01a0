"""Threads of the hierarchical far field's evaluation blocks (no GPU): for every
item size each target is stored by exactly one thread, the parts of a tile
are each taken once per target, and no working thread lacks a partner that
the reduction reads."""
import os
import subprocess

import pytest

SRC = r"""
#include <cstdio>
#include "tree.h"
using bie::tree::eval_slot;
int main() {
  for (int split = 0; split < 2; ++split) {
    const int nthreads = split ? 192 : 128;
    for (int nt = 1; nt <= 128; ++nt) {
      int writers[128] = {}, takers[128][8] = {};
      int parts = 0;
      for (int tid = 0; tid < nthreads; ++tid) {
        const auto s = eval_slot(nt, nthreads, split, tid);
        parts = s.parts;
        if (s.target < 0 || s.parts < 1 || s.parts > 8) return std::printf("slot %d %d\n", nt, tid), 1;
        if (s.writes) {
          if (s.target >= nt || !s.work) return std::printf("writer %d %d\n", nt, tid), 1;
          ++writers[s.target];
          // the reduction reads the other parts' threads at this stride
          for (int p = 1; p < s.parts; ++p) {
            const int o = tid + p * s.stride;
            if (o >= nthreads) return std::printf("partner %d %d\n", nt, tid), 1;
            const auto q = eval_slot(nt, nthreads, split, o);
            if (q.target != s.target || q.part != p || !q.work)
              return std::printf("partner %d %d\n", nt, tid), 1;
          }
        }
        if (s.work && s.target < nt) ++takers[s.target][s.part];
      }
      for (int t = 0; t < nt; ++t) {
        if (writers[t] != 1) return std::printf("%d writers of target %d of %d\n", writers[t], t, nt), 1;
        for (int p = 0; p < parts; ++p)
          if (takers[t][p] != 1) return std::printf("part %d of target %d of %d\n", p, t, nt), 1;
      }
    }
  }
  return 0;
}
"""


def test_one_writer_per_target(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src, exe = tmp_path / "slots.cpp", tmp_path / "slots"
    src.write_text(SRC)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I",
                    os.path.join(root, "fmm3dbie_b200", "csrc", "host"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("p", [4, 5, 6, 7, 8, 9, 11])
def test_repeated_products_are_identical(kind, p):
    """Grids whose last item leaves one to three spare warps: the sums have one
    writer and a fixed order, so repeated products are equal bit by bit."""
    import numpy as np
    import torch
    from fmm3dbie_b200 import Plan
    from fmm3dbie_b200 import surface as S
    s = S.torus_quad(14, 7, 4)
    zp = (2.0, -2.0j, 1.0) if kind else (1.0, 1.0)
    st = S.setup(s, kind, 1e-7, zp)
    P = Plan(kind, zp, s, st.near, st.over)
    x = np.random.default_rng(p).normal(size=s.npts)
    x = torch.tensor(x if kind == 0 else x * np.exp(1j * np.arange(s.npts)), device="cuda")
    for prec in (0, 1):
        P.set_far_method(prec, 1, 0.5, p, 64, 100)
        first = P.matvec(x, prec).clone()
        for _ in range(20):
            assert torch.equal(P.matvec(x, prec), first)
    P.close()
