// Multi-density far field of the FP32 path on the 5th-generation tensor cores.
//
// For nd densities the far field is, per target t and density m,
//   y(t, m) = sum_s K(t, s) sigma(s, m),
// a product of the kernel matrix with the density matrix.  Each CTA takes
// 128 targets, one source chunk and N densities and walks the chunk in tiles
// of 64 sources.  With K = Kr + i Ki and sigma = sr + i si (scaled by the
// source's weight / 4 pi) a tile adds
//   Re y += Kr sr - Ki si,   Im y += Kr si + Ki sr,
// formed as the two real products Kr [sr | si] and Ki [sr | si] in separate
// accumulators (one B operand for both, every MMA 2 N columns wide) and put
// together when they are read.  Every operand is split into high and low
// parts (x = hi + lo, both read as TF32), and the products lo*hi, hi*lo,
// hi*hi are issued in that order as tcgen05.mma kind::tf32 with FP32
// accumulators in tensor memory (the 3xTF32 scheme): an accumulator rounds
// after every K = 8 step, so the small products go in while it is small and
// only its last steps round at full size.
//
// The kernel values go from the registers that computed them straight into
// tensor memory (tcgen05.st, operand A); the density operand B is scaled,
// split and laid out once per matvec by far_tc_operand_kernel in the
// canonical no-swizzle K-major layout (8-row x 16-byte core matrices, row
// groups 128 B apart, K-direction core matrices (2 N / 8) x 128 B apart) and
// arrives by one bulk copy per tile.
//
// 18 warps per CTA, ordered only by mbarriers:
//   warps 0-15  kernel values (warp w: targets 32 (w % 4) .. + 31, one per
//               lane, sources 16 (w / 4) .. + 15 of the tile, two per packed
//               instruction) with the FP32 coordinates, block centring and
//               kernel of the CUDA-core kernels, whose rounding of a close
//               pair the error-matched W_eff32 fold cancels (the weight goes to
//               the density, so the values differ from theirs by roundings of
//               their own size); and the sums: each
//               thread adds N / 2 columns of its target into FP32 registers
//               after every tile and every kTcFold tiles into FP64 ones (64
//               densities: into FP32 sums in shared memory, compensated);
//   warp 16     producer: bulk copy of B, the tile's source coordinates;
//   warp 17     issues the MMAs (the warp runs uniformly, one elected lane
//               issues: from a single-lane branch the operands had to be
//               moved to uniform registers for each MMA, which took 9.3
//               instead of 5.7 ms at 16 densities).
// While the tensor core works on a tile the SIMT warps evaluate the next.
//
// Measured (matvec of a 36,504-node surface with 77,910 oversampled nodes,
// B200, against the kernel with serial stages or, up to 16 densities, the CUDA
// cores): 64 densities 17.3 -> 7.3 ms, 32: 15.5 -> 5.4, 16: 11.9 -> 5.0, 8: 8.4
// -> 5.0; at 4 both take 4.9 and the tuner keeps the CUDA cores.  Distance from
// the FP64 product there (k = 2, mean over plane waves): 64 densities 7.5e-7 ->
// 1.5e-7, 32: 7.5e-7 -> 1.3e-7, 16: 1.5e-7 -> 1.4e-7.  What bounds it: at 64
// densities the 48 MMAs of a tile (about 104 cycles each, 6.0 of the 7.3 ms; 64
// cycles would be the nominal rate) and the drain and the store of A between
// them, below that the kernel values with the operand splits (about 25
// instructions a pair; evaluation alone takes 3.4 of the 4.8 ms at 16).
//
// Completion waits are bounded (MatvecArgs::tc_spin polls); on timeout the
// kernel records the CTA in *err, every role leaves, the copies and MMAs in
// flight are waited for (bounded), the tensor memory is freed and the CTA's sums
// are NaN, so that no product goes on with what the buffer held before and a
// solve ends with a breakdown.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "device.cuh"
#include "pair.cuh"
#include "tc_common.cuh"

namespace bie {
namespace dev {
namespace {

constexpr int kTcT = 128;          // targets per CTA = accumulator rows
constexpr int kTcS = 64;           // sources per tile
constexpr int kTcWarps = 16;       // warps that evaluate kernel values
constexpr int kTcThreads = 32 * (kTcWarps + 2);
constexpr int kTcPer = kTcS * 4 / kTcWarps;  // sources of a tile per thread
constexpr int kTcFold = 8;         // tiles summed in the first set of registers
constexpr int kTcACols = 4 * kTcS; // tensor-memory columns of A: Kr hi, Ki hi, Kr lo, Ki lo
constexpr uint32_t kTcTmemCols = 512;

// Parts a tile's sources are split into for N densities: each part has its own
// two accumulators (Kr and Ki) of 2 N columns, so that an accumulator rounds
// at full size in 8 / parts hi*hi steps.  As many as tensor memory holds at 16
// densities (against FP64 on a 3,750-node sphere, without kTcLoss: 1.1e-7 with 4
// parts, 2.4e-7 with 1; the CUDA-core kernel 1.14e-7).
template <int N>
constexpr int kTcSplit = N == 64 ? 1 : (N == 32 ? 2 : 4);

// What an accumulator loses: it cuts to 24 bits after each K = 8 step, so a sum
// of n hi*hi steps comes out too small by about (n + 1) / 2 times the mean cut
// of one rounding toward zero (0.72 units of 2^-24 for mantissas spread as those
// of products are), more where the products themselves are cut to a large
// accumulator's last place.  Measured against the CUDA-core kernel, in units of
// 2^-24, on spheres, ellipsoids and tori of 864 to 36,504 nodes, k = 0.5 to 9 and
// complex, single and double layers and both, random densities (the low ends)
// and plane waves (the high ends): 2 steps 0.76 to 1.02, 4 steps 1.24 to 1.92,
// 8 steps 2.2 to 4.5.  The sums are scaled up by the middle of the range, so
// that what is left is below the CUDA-core kernel's own error (FP32 rsqrt, sine
// and cosine: -3 to +1 units); without it, plane waves of k = 0.5 on a
// 3,750-node sphere came out 1.4 times as far from FP64 as from that kernel.
template <int N>
constexpr double kTcLoss = (N == 64 ? 3.3 : N == 32 ? 1.6 : 0.9) / 16777216.0;

constexpr uint32_t kTcDrain = 1u << 22;  // polls of a wait for work in flight at the end
constexpr double kTcOver4Pi = 0.07957747154594767;
static_assert(kFarTileSources % kTcS == 0, "chunks are whole tiles");

// Floats of one tile's B operand (hi part, then lo part): 2 N rows (real
// parts, then imaginary parts of the densities) by kTcS sources.
template <int N>
constexpr int kTcOpFloats = 2 * 2 * N * kTcS;

// One tile's sources: coordinates negated and centred, normals.
struct TcGeom {
  float x[kTcS], y[kTcS], z[kTcS], nx[kTcS], ny[kTcS], nz[kTcS];
  int check, pad[3];
};

// Source tiles in flight; at 64 densities two, whose place the running sums
// take (a tile's MMAs take five times as long as its copy).
template <int N>
constexpr int kTcStages = N == 64 ? 2 : 3;

template <int N>
struct TcSmem {
  float b[kTcStages<N>][kTcOpFloats<N>];
  TcGeom geom[kTcStages<N>];
  float run[N == 64 ? 2 * N * 4 / kTcWarps : 1][N == 64 ? 32 * kTcWarps : 1];  // running sums
  uint64_t full[kTcStages<N>], empty[kTcStages<N>], afull, done;
  uint32_t tmem;
  int fail;
};

__device__ __forceinline__ bool tc_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Waits (at most `spin` polls) for phase `parity` of the barrier; false once any
// role of the CTA has given up.
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* fail,
                                        uint32_t spin) {
  for (uint32_t it = 0; it < spin; ++it) {
    if (tc_try(bar, parity)) return true;
    if (*fail) return false;
  }
  *fail = 1;
  return false;
}

// The same for a whole warp, one answer for all lanes.
__device__ __forceinline__ bool tc_wait_warp(uint64_t* bar, uint32_t parity, volatile int* fail,
                                             uint32_t spin) {
  return __all_sync(0xffffffffu, tc_wait(bar, parity, fail, spin));
}

__device__ __forceinline__ void tc_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Constants of the kernel values, each twice (the two lanes); a kernel
// parameter, so that they stay in the constant bank.
struct TcConst {
  float2 k, kim, ar, ai, br, bi, mbr, one, mone;
  float thr2;
  uint32_t spin;  // polls of a wait
};

// Kernel values K = alpha G + beta dG/dn of one target against two sources
// (lane .x and lane .y): the operations of pair_helm on the kernel's own constants
// in the place of a source's strengths.
template <bool CHECK, bool CK>
__device__ __forceinline__ void tc_pair(const float2 tx, const float2 ty, const float2 tz,
                                        const float2 msx, const float2 msy, const float2 msz,
                                        const float2 nx, const float2 ny, const float2 nz,
                                        const TcConst& c, float2& kr_, float2& ki_) {
  const float2 dx = __fadd2_rn(tx, msx), dy = __fadd2_rn(ty, msy), dz = __fadd2_rn(tz, msz);
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
  float2 rinv;
  rinv.x = (!CHECK || r2.x >= c.thr2) ? rsqrtf(r2.x) : 0.0f;
  rinv.y = (!CHECK || r2.y >= c.thr2) ? rsqrtf(r2.y) : 0.0f;
  const float2 r = __fmul2_rn(r2, rinv);
  const float2 kr = __fmul2_rn(c.k, r);
  float2 sn, cs;
  __sincosf(kr.x, &sn.x, &cs.x);
  __sincosf(kr.y, &sn.y, &cs.y);
  float2 rs = rinv;
  if (CK) {
    rs.x *= __expf(-c.kim.x * r.x);
    rs.y *= __expf(-c.kim.y * r.y);
  }
  const float2 dn = __ffma2_rn(dx, nx, __ffma2_rn(dy, ny, __fmul2_rn(dz, nz)));
  const float2 u = __fmul2_rn(dn, __fmul2_rn(rinv, rinv));
  float2 xr, xi;
  if (CK) {
    const float2 ur = __fmul2_rn(u, __ffma2_rn(c.kim, r, c.one));
    const float2 p = __fmul2_rn(u, kr);
    xr = __ffma2_rn(c.bi, p, __ffma2_rn(c.br, ur, c.ar));
    xi = __ffma2_rn(c.mbr, p, __ffma2_rn(c.bi, ur, c.ai));
  } else {
    xr = __ffma2_rn(u, __ffma2_rn(c.bi, kr, c.br), c.ar);
    xi = __ffma2_rn(u, __ffma2_rn(c.mbr, kr, c.bi), c.ai);
  }
  const float2 er = __fmul2_rn(xr, rs), ei = __fmul2_rn(xi, rs);
  const float2 msn = __fmul2_rn(sn, c.mone);
  kr_ = __ffma2_rn(cs, er, __fmul2_rn(msn, ei));
  ki_ = __ffma2_rn(cs, ei, __fmul2_rn(sn, er));
}

__device__ __forceinline__ void tmem_store16(uint32_t addr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16};" ::"r"(addr),
      "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]),
      "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
      : "memory");
}

// x -> high part (rounded to TF32) and remainder, which the tensor core reads
// as TF32 (of its 12 significant bits at most the last one goes, the size of a
// rounding of it; NaN for a NaN x).
__device__ __forceinline__ void split_store16(uint32_t hi_addr, uint32_t lo_addr, float* v) {
  float hi[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    hi[j] = tf32_rn(v[j]);
    v[j] -= hi[j];
  }
  tmem_store16(hi_addr, hi);
  tmem_store16(lo_addr, v);
}

__device__ __forceinline__ void tmem_load8(uint32_t addr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7])
               : "r"(addr));
}

// sum[n] += column c0 + n of Kr [sr | si] + i Ki [sr | si] from the tile's
// accumulators (this warp's lane quarter), two columns per packed operation:
// real parts Kr sr - Ki si, imaginary parts Kr si + Ki sr.
template <int N, int NH, int SPLIT>
__device__ __forceinline__ void flush_add(uint32_t tmem, int c0, float2* sum) {
  const bool re = c0 < N;
  const int ci = re ? c0 + N : c0 - N;
  const float2 sg = re ? make_float2(-1.f, -1.f) : make_float2(1.f, 1.f);
#pragma unroll
  for (int c = 0; c < NH; c += 8) {
    float v[SPLIT][2][8];
#pragma unroll
    for (int h = 0; h < SPLIT; ++h) {
      tmem_load8(tmem + uint32_t(h * 4 * N + c0 + c), v[h][0]);
      tmem_load8(tmem + uint32_t(h * 4 * N + 2 * N + ci + c), v[h][1]);
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float2 t[SPLIT];
#pragma unroll
      for (int h = 0; h < SPLIT; ++h)
        t[h] = __ffma2_rn(sg, make_float2(v[h][1][j], v[h][1][j + 1]),
                          make_float2(v[h][0][j], v[h][0][j + 1]));
      if constexpr (SPLIT >= 2) t[0] = __fadd2_rn(t[0], t[1]);
      if constexpr (SPLIT == 4) t[0] = __fadd2_rn(t[0], __fadd2_rn(t[2], t[3]));
      sum[(c + j) / 2] = __fadd2_rn(sum[(c + j) / 2], t[0]);
    }
  }
}

template <bool ACC>
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "n"(ACC ? 1 : 0)
      : "memory");
}

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.b32 %0, 1, 0, q;\n\t}\n"
      : "=r"(p));
  return p != 0;
}

// threadIdx.x, read anew.
__device__ __forceinline__ int fresh_tid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

template <int N, bool CK>
__global__ void __launch_bounds__(kTcThreads, 1)
    far_tc_kernel(const __grid_constant__ Geometry g, const __grid_constant__ TcConst c,
                  const float* __restrict__ ops, int64_t ntile_all, int nd,
                  double* __restrict__ partial, int64_t chunk_len, int* __restrict__ err) {
  constexpr int NB = 2 * N;               // accumulator columns: real, then imaginary parts
  constexpr int NH = NB * 4 / kTcWarps;   // of which each thread sums
  constexpr int SPLIT = kTcSplit<N>;
  static_assert(SPLIT * 2 * NB + kTcACols <= int(kTcTmemCols), "tensor memory");
  constexpr bool kTwoSums = N < 64;       // a second set of sums (64 densities: no registers left)
  constexpr int ST = kTcStages<N>;
  constexpr uint32_t kLboB = (NB / 8) * 128;
  constexpr uint32_t kOpBytes = kTcOpFloats<N> * sizeof(float);
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  TcSmem<N>& sm = *reinterpret_cast<TcSmem<N>*>(
      tc_smem + ((1024 - (smem_u32(tc_smem) & 1023)) & 1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t ntarg = g.ntarg, nptso = g.nptso;
  const int64_t tbase = int64_t(blockIdx.x) * kTcT;
  const int m0 = int(blockIdx.z) * N;
  // centre of the 512-target block, as the CUDA-core kernels and the fold use
  const int64_t tcen = (tbase / kFarBlockTargets32) * kFarBlockTargets32;
  const int64_t tcc = tcen < ntarg ? tcen : ntarg - 1;
  const double cx = g.tx[tcc], cy = g.ty[tcc], cz = g.tz[tcc];
  const int64_t s0 = int64_t(blockIdx.y) * chunk_len;
  const int64_t s1 = s0 + chunk_len < nptso ? s0 + chunk_len : nptso;
  const int ntiles = s1 > s0 ? int((s1 - s0 + kTcS - 1) / kTcS) : 0;

  if (warp == kTcWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&sm.tmem)),
                 "r"(kTcTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) {
    auto init = [](uint64_t* b, int n) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n));
    };
    for (int s = 0; s < ST; ++s) {
      init(&sm.full[s], 1);
      init(&sm.empty[s], kTcWarps + 1);
    }
    init(&sm.afull, kTcWarps);
    init(&sm.done, 1);
    sm.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem;
  const uint32_t acol = tmem + SPLIT * 2 * NB;  // A behind the accumulators
  volatile int* fail = &sm.fail;

  if (warp < kTcWarps) {
    const int quarter = warp & 3, sgrp = warp >> 2;
    const uint32_t lanes = uint32_t(quarter * 32) << 16;
    const int64_t it = tbase + 32 * quarter + lane;
    const int64_t ic = it < ntarg ? it : ntarg - 1;
    const float fx = float(g.tx[ic] - cx), fy = float(g.ty[ic] - cy), fz = float(g.tz[ic] - cz);
    const float2 tx = make_float2(fx, fx), ty = make_float2(fy, fy), tz = make_float2(fz, fz);
    const int c0 = sgrp * NH;  // this thread's accumulator columns
    float2 sum[NH / 2];
    double sum2[kTwoSums ? NH : 1];
#pragma unroll
    for (int n = 0; n < NH / 2; ++n) sum[n] = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = 0; n < NH; ++n) sum2[kTwoSums ? n : 0] = 0.0;
    bool ok = true;
    auto drain = [&](int i) {  // tile i's accumulator into the registers
      ok = tc_wait_warp(&sm.done, uint32_t(i) & 1u, fail, c.spin);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      flush_add<N, NH, SPLIT>(tmem + lanes, c0, sum);
      if (kTwoSums && i % kTcFold == kTcFold - 1) {
#pragma unroll
        for (int n = 0; n < NH / 2; ++n) {
          sum2[kTwoSums ? 2 * n : 0] += double(sum[n].x);
          sum2[kTwoSums ? 2 * n + 1 : 0] += double(sum[n].y);
          sum[n] = make_float2(0.f, 0.f);
        }
      }
    };
    // 64 densities: the sums so far into the running sums in shared memory; what
    // the addition rounds off (Knuth's TwoSum) starts the next sums, so that the
    // error does not grow with the number of tiles
    auto fold = [&]() {
#pragma unroll
      for (int n = 0; n < NH; ++n) {
        float& v = n & 1 ? sum[n / 2].y : sum[n / 2].x;
        float& r = sm.run[kTwoSums ? 0 : n][kTwoSums ? 0 : tid];
        const float a = r, t = __fadd_rn(a, v), b = __fsub_rn(t, a);
        v = __fadd_rn(__fsub_rn(a, __fsub_rn(t, b)), __fsub_rn(v, b));
        r = t;
      }
    };
    if (!kTwoSums)
#pragma unroll
      for (int n = 0; n < NH; ++n) sm.run[kTwoSums ? 0 : n][kTwoSums ? 0 : tid] = 0.f;
    const uint32_t a0 = acol + lanes + uint32_t(kTcPer * sgrp);
    for (int i = 0; i < ntiles; ++i) {
      const int s = i % ST;
      ok = tc_wait_warp(&sm.full[s], uint32_t(i / ST) & 1u, fail, c.spin);
      if (!ok) break;
      const TcGeom& ge = sm.geom[s];
      float vr[kTcPer], vi[kTcPer];
      auto eval = [&](auto chk) {
        constexpr bool C = decltype(chk)::value;
#pragma unroll
        for (int j = 0; j < kTcPer; j += 4) {
          const int q = kTcPer * sgrp + j;
          const float4 x = *reinterpret_cast<const float4*>(ge.x + q);
          const float4 y = *reinterpret_cast<const float4*>(ge.y + q);
          const float4 z = *reinterpret_cast<const float4*>(ge.z + q);
          const float4 nx = *reinterpret_cast<const float4*>(ge.nx + q);
          const float4 ny = *reinterpret_cast<const float4*>(ge.ny + q);
          const float4 nz = *reinterpret_cast<const float4*>(ge.nz + q);
          float2 a, b;
          tc_pair<C, CK>(tx, ty, tz, make_float2(x.x, x.y), make_float2(y.x, y.y),
                         make_float2(z.x, z.y), make_float2(nx.x, nx.y), make_float2(ny.x, ny.y),
                         make_float2(nz.x, nz.y), c, a, b);
          vr[j] = a.x, vr[j + 1] = a.y, vi[j] = b.x, vi[j + 1] = b.y;
          tc_pair<C, CK>(tx, ty, tz, make_float2(x.z, x.w), make_float2(y.z, y.w),
                         make_float2(z.z, z.w), make_float2(nx.z, nx.w), make_float2(ny.z, ny.w),
                         make_float2(nz.z, nz.w), c, a, b);
          vr[j + 2] = a.x, vr[j + 3] = a.y, vi[j + 2] = b.x, vi[j + 3] = b.y;
        }
      };
      if (ge.check)
        eval(std::true_type{});
      else
        eval(std::false_type{});
      __syncwarp();
      if (lane == 0) tc_arrive(&sm.empty[s]);
      // the tensor core is done with the previous tile's A and accumulators
      if (i > 0) {
        drain(i - 1);
        if (!ok) break;
      }
      split_store16(a0, a0 + 2 * kTcS, vr);
      split_store16(a0 + kTcS, a0 + 3 * kTcS, vi);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(&sm.afull);
      if (!kTwoSums && i > 0 && i % kTcFold == 0) fold();  // under this tile's MMAs
    }
    if (ok && ntiles > 0) drain(ntiles - 1);
    // (the indices are formed anew: kept over the loop they would be spilled)
    const int tid2 = fresh_tid(), c2 = (tid2 >> 7) * NH;
    const int64_t to = int64_t(blockIdx.x) * kTcT + (tid2 & (kTcT - 1));
    if (ok && to < ntarg) {
      // column c2 + n: real (< N) or imaginary part of density m0 + (c2 + n) % N
      const int comp = c2 >= N ? 1 : 0, d0 = int(blockIdx.z) * N + (c2 % N);
#pragma unroll
      for (int n = 0; n < NH; ++n)
        if (d0 + n < nd) {
          const double v = double(n & 1 ? sum[n / 2].y : sum[n / 2].x);
          partial[((size_t(blockIdx.y) * ntarg + to) * nd + d0 + n) * 2 + comp] =
              (1.0 + kTcLoss<N>) *
              (v + (kTwoSums ? sum2[kTwoSums ? n : 0]
                             : double(sm.run[kTwoSums ? 0 : n][kTwoSums ? 0 : tid2])));
        }
    }
  } else if (warp == kTcWarps) {
    // producer: lane j takes sources j, 32 + j of each tile.  The coordinates and the
    // bounding box of the next tile load while this one goes out.
    constexpr int H = kTcS / 32;
    const float* op = ops + (size_t(blockIdx.z) * ntile_all + size_t(s0 / kTcS)) * kTcOpFloats<N>;
    const double* tb = g.tbox && g.sbox ? g.tbox + 6 * (tbase / kFarBlockTargets32) : nullptr;
    double raw[H][6], sbx = 0.0;
    // lane d < 3: the target box's range in dimension d
    const double tlo = tb && lane < 3 ? tb[lane] : 0.0, thi = tb && lane < 3 ? tb[lane + 3] : 0.0;
    auto fetch = [&](int64_t sg) {  // the tile of sources from sg on
#pragma unroll
      for (int u = 0; u < H; ++u) {
        const int64_t s = sg + u * 32 + lane;
        const bool in = s < s1;
        // a padding source sits at the block centre: it keeps the threshold
        // test of its tile and meets zero densities
        raw[u][0] = in ? g.sx[s] : cx;
        raw[u][1] = in ? g.sy[s] : cy;
        raw[u][2] = in ? g.sz[s] : cz;
        raw[u][3] = in ? g.snx[s] : 0.0;
        raw[u][4] = in ? g.sny[s] : 0.0;
        raw[u][5] = in ? g.snz[s] : 0.0;
      }
      if (tb && lane < 6 && sg < s1) sbx = g.sbox[6 * (sg / kFarTileSources) + lane];
    };
    if (ntiles > 0) fetch(s0);
    int issued = 0;
    for (int i = 0; i < ntiles; ++i) {
      const int s = i % ST;
      const int64_t sg = s0 + int64_t(i) * kTcS;
      float cur[H][6];
#pragma unroll
      for (int u = 0; u < H; ++u) {
        cur[u][0] = -float(raw[u][0] - cx);
        cur[u][1] = -float(raw[u][1] - cy);
        cur[u][2] = -float(raw[u][2] - cz);
#pragma unroll
        for (int d = 3; d < 6; ++d) cur[u][d] = float(raw[u][d]);
      }
      const double shi = __shfl_down_sync(0xffffffffu, sbx, 3);
      const double gap = lane < 3 ? fmax(fmax(sbx - thi, tlo - shi), 0.0) : 0.0;
      const double g2 = gap * gap;
      const double gap2 = g2 + __shfl_down_sync(0xffffffffu, g2, 1) + __shfl_down_sync(0xffffffffu, g2, 2);
      if (i + 1 < ntiles) fetch(sg + kTcS);
      if (i >= ST && !tc_wait_warp(&sm.empty[s], uint32_t(i / ST - 1) & 1u, fail, c.spin)) break;
      TcGeom& ge = sm.geom[s];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int j = 32 * h + lane;
        ge.x[j] = cur[h][0];
        ge.y[j] = cur[h][1];
        ge.z[j] = cur[h][2];
        ge.nx[j] = cur[h][3];
        ge.ny[j] = cur[h][4];
        ge.nz[j] = cur[h][5];
      }
      // only a whole tile may skip the threshold test (padding needs it)
      if (lane == 0) ge.check = !tb || sg + kTcS > s1 || gap2 <= g.box_margin2;
      __syncwarp();
      if (lane == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                         smem_u32(&sm.full[s])),
                     "r"(kOpBytes)
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(smem_u32(sm.b[s])),
            "l"(op + size_t(i) * kTcOpFloats<N>), "r"(kOpBytes), "r"(smem_u32(&sm.full[s]))
            : "memory");
      }
      issued = i + 1;
    }
    // the copies still in flight land before the CTA goes: another role may give
    // up after this one has left its loop
    for (int i = issued > ST ? issued - ST : 0; i < issued; ++i)
      for (uint32_t r = 0; r < kTcDrain; ++r)
        if (tc_try(&sm.full[i % ST], uint32_t(i / ST) & 1u)) break;
  } else {
    // the whole warp walks the tiles, so that the operands of the MMAs stay
    // in uniform registers; one elected lane issues
    constexpr uint32_t kAll = idesc_tf32(kTcT, NB);
    const uint64_t bdesc = smem_desc(smem_u32(sm.b[0]), kLboB);
    int issued = -1;
    for (int i = 0; i < ntiles; ++i) {
      const int s = i % ST;
      if (!tc_wait_warp(&sm.full[s], uint32_t(i / ST) & 1u, fail, c.spin)) break;
      if (!tc_wait_warp(&sm.afull, uint32_t(i) & 1u, fail, c.spin)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t bd = bdesc + uint64_t(uint32_t(s) * (kOpBytes >> 4));
      if (elect_one()) {
        // lo*hi, hi*lo, hi*hi
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          const uint32_t ap = acol + (p == 0 ? 2 * kTcS : 0);
          const uint64_t bp = bd + (p == 1 ? uint64_t(kOpBytes / 2) >> 4 : 0);
#pragma unroll
          for (int ks = 0; ks < kTcS / 8; ++ks) {
            const uint64_t bk = bp + uint64_t((ks * 2 * kLboB) >> 4);
            constexpr int per = kTcS / 8 / SPLIT;
            const uint32_t d = tmem + uint32_t(ks / per) * 2 * NB;
            if (p == 0 && ks % per == 0) {
              tc_mma<false>(d, ap + 8 * ks, bk, kAll);
              tc_mma<false>(d + NB, ap + kTcS + 8 * ks, bk, kAll);
            } else {
              tc_mma<true>(d, ap + 8 * ks, bk, kAll);
              tc_mma<true>(d + NB, ap + kTcS + 8 * ks, bk, kAll);
            }
          }
        }
        tc_commit(&sm.empty[s]);  // (first: nobody waits for the last tile's)
        tc_commit(&sm.done);
      }
      __syncwarp();
      issued = i;
    }
    // the last committed MMAs finish before the tensor memory is freed
    for (uint32_t r = 0; issued >= 0 && r < kTcDrain; ++r)
      if (tc_try(&sm.done, uint32_t(issued) & 1u)) break;
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*fail) {
    if (tid == 0 && err) atomicExch(err, 1 + int(blockIdx.x));
    for (int q = fresh_tid(); q < kTcT * N; q += kTcThreads) {
      const int64_t to = int64_t(blockIdx.x) * kTcT + q / N;
      const int m = int(blockIdx.z) * N + q % N;
      if (to < ntarg && m < nd)
        reinterpret_cast<double2*>(partial)[(size_t(blockIdx.y) * ntarg + to) * nd + m] =
            make_double2(CUDART_NAN, CUDART_NAN);
    }
  }
  if (warp == kTcWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTcTmemCols));
}

// B operand of every tile: the oversampled densities times weight / 4 pi,
// split into high and low parts, rows real then imaginary, zero beyond the
// last source and density.  One block per (tile, density group, quarter of the
// tile's sources): with one block a tile a surface of 864 nodes waited 5 to 9 us
// for 50 blocks.
constexpr int kTcOpParts = 4;

template <int N>
__global__ void far_tc_operand_kernel(Geometry g, const float* __restrict__ sig, int nd,
                                      float* __restrict__ ops) {
  constexpr uint32_t kLboB = (2 * N / 8) * 128;
  constexpr int PS = kTcS / kTcOpParts;
  static_assert(PS % 4 == 0, "whole groups of four sources");
  const int64_t tile = blockIdx.x;
  const int p0 = int(blockIdx.z) * PS;  // first source of this block in the tile
  const int64_t sb = tile * kTcS + p0;
  const int m0 = int(blockIdx.y) * N;
  __shared__ float sv[PS][2 * N + 1];
  for (int q = threadIdx.x; q < PS * N; q += blockDim.x) {
    const int j = q / N, m = q - j * N;
    const int64_t s = sb + j;
    float2 v = make_float2(0.f, 0.f);
    if (s < g.nptso && m0 + m < nd) {
      const double f = g.sw[s] * kTcOver4Pi;
      const float2 u = reinterpret_cast<const float2*>(sig)[size_t(s) * nd + m0 + m];
      v = make_float2(float(double(u.x) * f), float(double(u.y) * f));
    }
    sv[j][m] = v.x;
    sv[j][N + m] = v.y;
  }
  __syncthreads();
  float* hi = ops + (size_t(blockIdx.y) * gridDim.x + tile) * kTcOpFloats<N>;
  float* lo = hi + kTcOpFloats<N> / 2;
  for (int q = threadIdx.x; q < 2 * N * (PS / 4); q += blockDim.x) {
    const int r = q % (2 * N), k = 4 * (q / (2 * N));
    store_split(hi, lo, op_off(r, p0 + k, kLboB), sv[k][r], sv[k + 1][r], sv[k + 2][r],
                sv[k + 3][r]);
  }
}

template <int N, bool CK>
cudaError_t far_tc_go(const Geometry& g, const KParams& kp, const MatvecArgs& a, cudaStream_t st,
                      int* occ) {
  auto kern = far_tc_kernel<N, CK>;
  const size_t smem = sizeof(TcSmem<N>) + 1024;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(smem));
  if (e != cudaSuccess) return e;
  if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, kTcThreads, smem);
  if (!a.tc_ops) return cudaErrorInvalidValue;
  const int64_t tblocks = (g.ntarg + kTcT - 1) / kTcT;
  const int groups = (a.nd + N - 1) / N;
  const int64_t ntile = (g.nptso + kTcS - 1) / kTcS;
  int64_t chunk = (g.nptso + a.nchunks - 1) / a.nchunks;
  chunk = ((chunk + kFarTileSources - 1) / kFarTileSources) * kFarTileSources;
  far_tc_operand_kernel<N><<<dim3(unsigned(ntile), unsigned(groups), kTcOpParts), 256, 0, st>>>(
      g, static_cast<const float*>(a.strengths), a.nd, a.tc_ops);
  note_launches(1);
  const dim3 grid(unsigned(tblocks), unsigned(a.nchunks), unsigned(groups));
  auto dup = [](double v) { return make_float2(float(v), float(v)); };
  TcConst c;
  c.k = dup(kp.kr);
  c.kim = dup(kp.ki);
  c.ar = dup(kp.ar);
  c.ai = dup(kp.ai);
  c.br = dup(kp.br);
  c.bi = dup(kp.bi);
  c.mbr = dup(-kp.br);
  c.one = dup(1.0);
  c.mone = dup(-1.0);
  c.thr2 = float(kp.thresh * kp.thresh);
  c.spin = a.tc_spin;
  kern<<<grid, kTcThreads, smem, st>>>(g, c, a.tc_ops, ntile, a.nd, a.partial, chunk, a.tc_err);
  return cudaGetLastError();
}

template <int N>
cudaError_t far_tc_n(const Geometry& g, const KParams& kp, const MatvecArgs& a, cudaStream_t st,
                     int* occ) {
  return kp.ki != 0.0 ? far_tc_go<N, true>(g, kp, a, st, occ)
                      : far_tc_go<N, false>(g, kp, a, st, occ);
}

}  // namespace

int far_tc_targets(int precision) { return precision == 1 ? kTcT : far_dmma_targets(); }

int far_tc_group(int variant, int nd, int precision, int kind) {
  if (variant < 3 || variant > 4 || kind != 1) return 0;
  if (precision == 0) {
    // FP64: from 9 densities, where the CUDA-core kernel holds fewer than a
    // block here (at 4 and 8 the padding to 16 columns costs more)
    if (variant == 4) return nd > 32 ? 32 : 0;
    return nd <= 8 ? 0 : nd <= 16 ? 16 : nd <= 32 ? 32 : 64;
  }
  if (nd < 2) return 0;
  if (variant == 4) return nd > 32 ? 64 : 0;
  return nd <= 16 ? 16 : 32;
}

size_t far_tc_operand_floats(int nd, int precision, int kind, int64_t nptso) {
  size_t most = 0;
  if (precision != 1) return 0;
  for (int v = 3; v <= 4; ++v) {
    const int n = far_tc_group(v, nd, precision, kind);
    if (n > 0) most = std::max(most, size_t((nd + n - 1) / n) * n);
  }
  return most * size_t((nptso + kTcS - 1) / kTcS) * (2 * 2 * kTcS);
}

cudaError_t far_tc(int variant, const Geometry& g, const KParams& kp, const MatvecArgs& a,
                   cudaStream_t st, int* occ) {
  const int group = far_tc_group(variant, a.nd, a.precision, kp.kind);
  if (group > 0 && a.precision == 0) return far_dmma(group, g, kp, a, st, occ);
  switch (group) {
    case 16:
      return far_tc_n<16>(g, kp, a, st, occ);
    case 32:
      return far_tc_n<32>(g, kp, a, st, occ);
    case 64:
      return far_tc_n<64>(g, kp, a, st, occ);
    default:
      if (occ) *occ = 0;
      return cudaErrorInvalidValue;
  }
}

}  // namespace dev
}  // namespace bie
