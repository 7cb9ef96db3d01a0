// Evaluation of one shared-memory tile of sources against one target per
// thread: the hierarchical far field's lists and the direct far field of small
// problems.
#pragma once
#include <cuda_runtime.h>

#include "pair.cuh"

namespace bie {
namespace dev {
namespace {

// A tile in shared memory.  FP32: one array per value, the coordinates
// negated, so that a thread reads four consecutive sources at a time and
// evaluates two per packed instruction; FP64: one record per source.
template <int KIND, typename R, int TILE>
struct TileSmem {
  double4 g0[TILE];
  double2 g1[TILE];
  double4 st[TILE];
};
template <int KIND, int TILE>
struct TileSmem<KIND, float, TILE> {
  float v[KIND == 1 ? 10 : 8][TILE];  // x, y, z, nx, ny, nz, charge, dipole
};

// FP32: the tile's sources j0 .. j1 - 1 (a multiple of 4; sources past the
// tile's end carry no strength) against one target, two per packed
// instruction, two at a time; per lane the operations of pair_helm,
// pair_lap and pair_charge.
template <int KIND, bool CK, int MODE, int TILE>  // MODE: entry kind
__device__ __forceinline__ void tile_eval(const TileSmem<KIND, float, TILE>& T, int j0, int j1,
                                          float tx, float ty, float tz, float k, float kim,
                                          float thr2, float& outr, float& outi) {
  const float2 x = make_float2(tx, tx), y = make_float2(ty, ty), z = make_float2(tz, tz);
  const float2 k2 = make_float2(k, k), kim2 = make_float2(kim, kim);
  float2 pa = make_float2(0.f, 0.f), pb = pa, pi = pa;
  auto at = [&](int a, int j) { return *reinterpret_cast<const float4*>(&T.v[a][j]); };
  auto lo = [](const float4& q) { return make_float2(q.x, q.y); };
  auto hi = [](const float4& q) { return make_float2(q.z, q.w); };
  auto charge = [&](float2 sx, float2 sy, float2 sz, float2 cr, float2 ci) {
    const float2 dx = __fadd2_rn(x, sx), dy = __fadd2_rn(y, sy), dz = __fadd2_rn(z, sz);
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    float2 rinv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
    if constexpr (KIND == 1) {
      const float2 r = __fmul2_rn(r2, rinv), kr = __fmul2_rn(k2, r);
      float2 sn, cs;
      __sincosf(kr.x, &sn.x, &cs.x);
      __sincosf(kr.y, &sn.y, &cs.y);
      if (CK) {
        rinv.x *= __expf(-kim * r.x);
        rinv.y *= __expf(-kim * r.y);
      }
      const float2 er = __fmul2_rn(cr, rinv), ei = __fmul2_rn(ci, rinv);
      pa = __ffma2_rn(cs, er, pa);
      pb = __ffma2_rn(sn, ei, pb);
      pi = __ffma2_rn(cs, ei, __ffma2_rn(sn, er, pi));
    } else {
      pa = __ffma2_rn(cr, rinv, pa);
    }
  };
#pragma unroll 2
  for (int j = j0; j < j1; j += 4) {
    const float4 sx = at(0, j), sy = at(1, j), sz = at(2, j);
    if constexpr (MODE == 2) {
      const float4 cr = at(6, j), ci = KIND == 1 ? at(7, j) : cr;
      charge(lo(sx), lo(sy), lo(sz), lo(cr), lo(ci));
      charge(hi(sx), hi(sy), hi(sz), hi(cr), hi(ci));
    } else {
      const float4 nx = at(3, j), ny = at(4, j), nz = at(5, j);
      if constexpr (KIND == 1) {
        const float4 cr = at(6, j), ci = at(7, j), dr = at(8, j), di = at(9, j);
        const float4 md = make_float4(-dr.x, -dr.y, -dr.z, -dr.w);
        pair_helm_x2<MODE == 0>(x, y, z, lo(sx), lo(sy), lo(sz), lo(nx), lo(ny), lo(nz), lo(cr),
                                lo(ci), lo(dr), lo(di), lo(md), k2, kim2, thr2, CK, pa, pb, pi);
        pair_helm_x2<MODE == 0>(x, y, z, hi(sx), hi(sy), hi(sz), hi(nx), hi(ny), hi(nz), hi(cr),
                                hi(ci), hi(dr), hi(di), hi(md), k2, kim2, thr2, CK, pa, pb, pi);
      } else {
        const float4 c = at(6, j), d = at(7, j);
        pair_lap_x2<MODE == 0>(x, y, z, lo(sx), lo(sy), lo(sz), lo(nx), lo(ny), lo(nz), lo(c),
                               lo(d), thr2, pa);
        pair_lap_x2<MODE == 0>(x, y, z, hi(sx), hi(sy), hi(sz), hi(nx), hi(ny), hi(nz), hi(c),
                               hi(d), thr2, pa);
      }
    }
  }
  outr = (pa.x - pb.x) + (pa.y - pb.y);
  outi = pi.x + pi.y;
}

template <int KIND, bool CK, int MODE, int TILE>
__device__ __forceinline__ void tile_eval(const TileSmem<KIND, double, TILE>& T, int j0, int j1,
                                          double tx, double ty, double tz, double k, double kim,
                                          double thr2, double& outr, double& outi,
                                          const double2* tab) {
  outr = outi = 0.0;
#pragma unroll 4
  for (int j = j0; j < j1; ++j) {
    const double4 s = T.st[j];
    if constexpr (MODE == 2)
      pair_charge<KIND>(tx, ty, tz, T.g0[j], s, k, kim, CK, outr, outi, tab);
    else if constexpr (KIND == 1)
      pair_helm<MODE == 0>(tx, ty, tz, T.g0[j], T.g1[j], s, k, kim, thr2, CK, outr, outi, tab);
    else
      pair_lap<double, MODE == 0>(tx, ty, tz, T.g0[j], T.g1[j], make_double2(s.x, s.y), thr2, outr);
  }
}

// Stores source q of a tile (coordinates less the centre c, rounded to R; s:
// charge and dipole strengths or a proxy charge).
template <int KIND, typename R, int TILE>
__device__ __forceinline__ void tile_store(TileSmem<KIND, R, TILE>& T, int q, double x, double y,
                                           double z, double nx, double ny, double nz, double cx,
                                           double cy, double cz, typename Vec<R>::T4 s) {
  if constexpr (sizeof(R) == 4) {
    T.v[0][q] = -R(x - cx);
    T.v[1][q] = -R(y - cy);
    T.v[2][q] = -R(z - cz);
    T.v[3][q] = R(nx);
    T.v[4][q] = R(ny);
    T.v[5][q] = R(nz);
    T.v[6][q] = s.x;
    T.v[7][q] = s.y;
    if constexpr (KIND == 1) {
      T.v[8][q] = s.z;
      T.v[9][q] = s.w;
    }
  } else {
    (void)cx, (void)cy, (void)cz;
    T.g0[q] = make_double4(x, y, z, nx);
    T.g1[q] = make_double2(ny, nz);
    T.st[q] = s;
  }
}

}  // namespace
}  // namespace dev
}  // namespace bie
