// Table-driven FP64 sine and cosine shared by the far-field and
// near-quadrature kernels.
#pragma once

namespace bie {
namespace dev {

// Table-driven sine and cosine (FP64) (the table-driven
// reduction of P. T. P. Tang, ACM TOMS 15 (1989) / 16 (1990)):
//   x = j (2 pi / N) + rho,  |rho| <= pi / N,
//   sin x = S_j cos rho + C_j sin rho,  cos x = C_j cos rho - S_j sin rho,
// with (C_j, S_j) = (cos, sin)(2 pi j / N) from a per-block table and the
// Taylor series of sin rho (to rho^5) and cos rho (to rho^6), whose first
// omitted terms are below 1e-17 for |rho| <= pi/256.  2 pi / N is split as
// C1 + C2 with C1 rounded to 24 bits, so j C1 is exact for |j| < 2^29.
constexpr int kTrigN = 256;
constexpr double kTrigStep = 0.02454369260617026;     // 2 pi / 256
constexpr double kTrigInvStep = 40.74366543152521;    // 256 / (2 pi)
constexpr double kTrigC1 = 0.02454369328916073;       // float(2 pi / 256)
constexpr double kTrigC2 = -6.829904687791004e-10;    // 2 pi / 256 - C1

// Fills tab[q] = (cos, sin)(2 pi q / N) with the block's threads.
__device__ __forceinline__ void fill_trig_table(double2* tab) {
  for (int q = threadIdx.x; q < kTrigN; q += blockDim.x) {
    double sq, cq;
    sincos(double(q) * kTrigStep, &sq, &cq);
    tab[q] = make_double2(cq, sq);
  }
}

__device__ __forceinline__ void sincos_tab(double x, const double2* tab, double& s, double& c) {
  const double jd = rint(x * kTrigInvStep);
  const int j = int(jd) & (kTrigN - 1);
  double rho = fma(-jd, kTrigC1, x);
  rho = fma(-jd, kTrigC2, rho);
  const double r2 = rho * rho;
  const double sp = fma(rho * r2, fma(r2, 1.0 / 120.0, -1.0 / 6.0), rho);
  const double cp = fma(r2, fma(r2, fma(r2, -1.0 / 720.0, 1.0 / 24.0), -0.5), 1.0);
  const double2 t = tab[j];
  s = fma(t.y, cp, t.x * sp);
  c = fma(t.x, cp, -(t.y * sp));
}

// The far-field variant of the same method, for the direct and hierarchical
// far-field kernels, whose phases k r stay below a few hundred (the surface in
// wavelengths times 2 pi).  The FP64 pipe bounds those kernels, so the table is
// fine enough for short series and nothing is converted:
//   j = rint(x N / (2 pi)) by adding 1.5 * 2^52 (no conversion instructions),
//   rho = x - j (2 pi / N) in one fused multiply-add with 2 pi / N rounded to
//   FP64 (relative error 3.9e-17: the phase is off by as much of itself, a
//   third of the rounding of k r),
//   sin rho to rho^5 and cos rho to rho^4, |rho| <= pi / 1024: next terms
//   rho^7 / 5040 = 5e-22 and rho^6 / 720 = 1.2e-18.
// 13 FP64 operations; 256 entries took 15.  Distance of (sin, cos) from the true
// values of k r: 2.0e-16 at most for phases up to 1 (256 entries: 2.4e-16), and
// otherwise the rounding of k r, as there: 1.1e-14 up to 100.  (With the phase
// taken straight to table steps, x = r (k N / (2 pi)), and a two-term sine it
// was 12 operations, but 3.6e-16 up to 1, and the rounding of k N / (2 pi) moved
// the whole wavenumber by up to 1.7e-16 of itself.)
constexpr int kFarTrigN = 1024;
constexpr double kFarTrigInvStep = 162.97466172610083;  // 1024 / (2 pi)
constexpr double kFarTrigStep = 0.006135923151542565;   // 2 pi / 1024
constexpr double kRoundMagic = 6755399441055744.0;      // 1.5 * 2^52

// Fills tab[q] = (cos, sin)(2 pi q / N): the first octant by sincos (one
// value a thread for 128 threads), the others by symmetry.  Ends with a
// barrier.
__device__ __forceinline__ void fill_far_trig_table(double2* tab) {
  constexpr int E = kFarTrigN / 8;
  for (int q = threadIdx.x; q <= E; q += blockDim.x) {
    double s, c;
    sincospi(double(q) / (kFarTrigN / 2), &s, &c);
    tab[q] = make_double2(c, s);
  }
  __syncthreads();
  for (int q = E + 1 + threadIdx.x; q < kFarTrigN; q += blockDim.x) {
    const int o = q / E, r = q % E;
    const double2 t = tab[o & 1 ? E - r : r];  // entries 0 .. E only
    const double c = o & 1 ? t.y : t.x, s = o & 1 ? t.x : t.y;  // within the quadrant
    const int quad = o >> 1;
    tab[q] = quad == 0   ? make_double2(c, s)
             : quad == 1 ? make_double2(-s, c)
             : quad == 2 ? make_double2(-c, -s)
                         : make_double2(s, -c);
  }
  __syncthreads();
}

__device__ __forceinline__ void sincos_far(double x, const double2* tab, double& s, double& c) {
  const double u = fma(x, kFarTrigInvStep, kRoundMagic);
  const int j = __double2loint(u) & (kFarTrigN - 1);
  const double rho = fma(kRoundMagic - u, kFarTrigStep, x);
  const double r2 = rho * rho;
  const double sp = fma(rho * r2, fma(r2, 1.0 / 120.0, -1.0 / 6.0), rho);
  const double cp = fma(r2, fma(r2, 1.0 / 24.0, -0.5), 1.0);
  const double2 t = tab[j];
  s = fma(t.y, cp, t.x * sp);
  c = fma(t.x, cp, -(t.y * sp));
}

// 1/sqrt(a) in FP64 for normal a > 0: the hardware's FP64 approximation y0
// (rsqrt.approx.ftz.f64, relative error e0 / 2 with e0 = 1 - a y0^2 about
// 2^-20) refined by one third-order step of the binomial series of
// (1 - e)^(-1/2):
//   y = y0 (1 + e/2 + 3 e^2 / 8),
// whose truncation error 5 e^3 / 16 is below the FP64 rounding.  Starting
// from the FP32 approximation took two conversions more, on the pipe that
// the approximation itself uses.
__device__ __forceinline__ double rsqrt_far(double a) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(a));
  const double e = fma(-(a * y0), y0, 1.0);
  return fma(y0 * e, fma(e, 0.375, 0.5), y0);
}

}  // namespace dev
}  // namespace bie
