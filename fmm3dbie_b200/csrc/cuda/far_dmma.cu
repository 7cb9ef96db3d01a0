// Multi-density far field of the FP64 Helmholtz path with FP64 matrix
// instructions (mma.sync.m8n8k4.f64; the 5th-generation tensor cores have no
// FP64 kind).
//
// The far field of nd densities is the product of the kernel matrix with the
// density matrix.  A warp takes 16 targets (two row tiles of 8) and all N
// densities of its block: per step of 4 sources lane (row, source) = (lane / 4,
// lane % 4) evaluates the kernel value K of its two targets against its
// source, which is exactly its element of the matrix instruction's A operand;
// the densities of the 4 sources come from shared memory as B operands (one
// 16-byte load holds the real and the imaginary one) and serve both row tiles:
//   Re y += Kr sr - Ki si,   Im y += Kr si + Ki sr
// in FP64 accumulators kept in registers over the whole chunk.
//
// The CUDA-core kernel (far_md_kernel) holds 16 densities a thread and so
// evaluates every kernel value four times at 64 densities (424 operations a
// pair against 298 here), with one instruction per multiply-add; a matrix
// instruction is 256 of them.  Both are bound by the FP64 pipe (here 90 % busy,
// 77 % of it with matrix instructions).  36,504 targets x 77,910 sources: 64
// densities 86.3 -> 52.5 ms (47 ms at the pipe's peak), 24 densities 44.4 ->
// 30.2, 16 densities 22.8 -> 19.1.
#include <cuda_runtime.h>

#include <cstdint>

#include "device.cuh"
#include "pair.cuh"

namespace bie {
namespace dev {
namespace {

constexpr int kDmThreads = 128;
constexpr int kDmT = 16 * (kDmThreads / 32);  // targets per block
constexpr int kDmS = 32;                      // sources per tile
static_assert(kFarTileSources % kDmS == 0, "chunks are whole tiles");

template <int N>
struct DmSmem {
  double2 sig[2][kDmS][N + 2];  // the pad spreads a step's 4 sources over the banks
  double4 g0[2][kDmS], ab[2][kDmS];
  double2 g1[2][kDmS];
  double2 trig[kFarTrigN];
};

__device__ __forceinline__ void dmma(double* c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

template <int N, bool CK>
__global__ void __launch_bounds__(kDmThreads, N == 64 ? 2 : 3)
    far_dmma_kernel(Geometry g, KParams kp, const double4* __restrict__ ab,
                    const double2* __restrict__ sig, int nd, double2* __restrict__ partial,
                    int64_t chunk_len) {
  extern __shared__ __align__(16) unsigned char dm_smem[];
  DmSmem<N>& sm = *reinterpret_cast<DmSmem<N>*>(dm_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = lane >> 2, src = lane & 3;
  const int m0 = int(blockIdx.z) * N;
  fill_far_trig_table(sm.trig);
  const int64_t t0 = int64_t(blockIdx.x) * kDmT + 16 * warp + row;
  double tx[2], ty[2], tz[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int64_t it = t0 + 8 * u < g.ntarg ? t0 + 8 * u : g.ntarg - 1;
    tx[u] = g.tx[it];
    ty[u] = g.ty[it];
    tz[u] = g.tz[it];
  }
  const double thr2 = kp.thresh * kp.thresh;
  const int64_t s0 = int64_t(blockIdx.y) * chunk_len;
  const int64_t s1 = s0 + chunk_len < g.nptso ? s0 + chunk_len : g.nptso;
  // tile of sources from sb on into buffer b: densities as asynchronous
  // copies (zeros past the last source or density), geometry by plain loads
  auto load = [&](int64_t sb, int b) {
    for (int q = tid; q < kDmS * N; q += kDmThreads) {
      const int j = q / N, m = q - j * N;
      const bool in = sb + j < s1 && m0 + m < nd;
      const double2* from = sig + (in ? size_t(sb + j) * nd + m0 + m : 0);
      const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(&sm.sig[b][j][m]));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(from),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (tid < kDmS) {
      const int64_t s = sb + tid;
      const double4 z = make_double4(0.0, 0.0, 0.0, 0.0);
      const bool in = s < s1;
      sm.g0[b][tid] = in ? make_double4(g.sx[s], g.sy[s], g.sz[s], g.snx[s]) : z;
      sm.g1[b][tid] = in ? make_double2(g.sny[s], g.snz[s]) : make_double2(0.0, 0.0);
      sm.ab[b][tid] = in ? ab[s] : z;
    }
  };
  double re[2][N / 8][2], im[2][N / 8][2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int j = 0; j < N / 8; ++j) re[u][j][0] = re[u][j][1] = im[u][j][0] = im[u][j][1] = 0.0;
  if (s0 < s1) load(s0, 0);
  int b = 0;
  for (int64_t sb = s0; sb < s1; sb += kDmS, b ^= 1) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // this tile has landed, and every warp is done with the other buffer
    if (sb + kDmS < s1) load(sb + kDmS, b ^ 1);
#pragma unroll 1
    for (int st = 0; st < kDmS; st += 4) {
      const int s = st + src;
      const double4 a = sm.g0[b][s], w = sm.ab[b][s];
      const double2 n = sm.g1[b][s];
      double kr[2], ki[2], mi[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        kr[u] = ki[u] = 0.0;
        pair_helm(tx[u], ty[u], tz[u], a, n, w, kp.kr, kp.ki, thr2, CK, kr[u], ki[u], sm.trig);
        mi[u] = -ki[u];
      }
#pragma unroll
      for (int j = 0; j < N / 8; ++j) {
        const double2 d = sm.sig[b][s][8 * j + row];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          dmma(re[u][j], kr[u], d.x);
          dmma(im[u][j], kr[u], d.y);
          dmma(re[u][j], mi[u], d.y);
          dmma(im[u][j], ki[u], d.x);
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int64_t it = t0 + 8 * u;
    if (it >= g.ntarg) continue;
#pragma unroll
    for (int j = 0; j < N / 8; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int m = m0 + 8 * j + 2 * src + c;
        if (m < nd)
          partial[(size_t(blockIdx.y) * g.ntarg + it) * nd + m] = make_double2(re[u][j][c], im[u][j][c]);
      }
  }
}

template <int N, bool CK>
cudaError_t far_dmma_go(const Geometry& g, const KParams& kp, const MatvecArgs& a,
                        cudaStream_t st, int* occ) {
  auto kern = far_dmma_kernel<N, CK>;
  const size_t smem = sizeof(DmSmem<N>);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, kDmThreads, smem);
  const int64_t tblocks = (g.ntarg + kDmT - 1) / kDmT;
  const int groups = (a.nd + N - 1) / N;
  int64_t chunk = (g.nptso + a.nchunks - 1) / a.nchunks;
  chunk = ((chunk + kFarTileSources - 1) / kFarTileSources) * kFarTileSources;
  kern<<<dim3(unsigned(tblocks), unsigned(a.nchunks), unsigned(groups)), kDmThreads, smem, st>>>(
      g, kp, static_cast<const double4*>(a.ab), static_cast<const double2*>(a.strengths), a.nd,
      reinterpret_cast<double2*>(a.partial), chunk);
  return cudaGetLastError();
}

template <int N>
cudaError_t far_dmma_n(const Geometry& g, const KParams& kp, const MatvecArgs& a, cudaStream_t st,
                       int* occ) {
  return kp.ki != 0.0 ? far_dmma_go<N, true>(g, kp, a, st, occ)
                      : far_dmma_go<N, false>(g, kp, a, st, occ);
}

}  // namespace

int far_dmma_targets() { return kDmT; }

cudaError_t far_dmma(int group, const Geometry& g, const KParams& kp, const MatvecArgs& a,
                     cudaStream_t st, int* occ) {
  switch (group) {
    case 16:
      return far_dmma_n<16>(g, kp, a, st, occ);
    case 32:
      return far_dmma_n<32>(g, kp, a, st, occ);
    default:
      return far_dmma_n<64>(g, kp, a, st, occ);
  }
}

}  // namespace dev
}  // namespace bie
