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
// far-field kernels, whose phases stay below 100 and whose products only need
// ~1e-14.  The FP64 pipe bounds those kernels, so the phase goes straight to
// table steps and the table is fine enough for short series:
//   u = k r N / (2 pi) = j + f, |f| <= 1/2, j by the round-to-integer of adding
//   1.5 * 2^52 (no conversion instructions), f = u - j in one fused
//   multiply-add (its error is the rounding of k N / (2 pi): 1.1e-16 of the
//   phase);
//   sin(2 pi f / N) to f^3, with the f^5 term economised on |f| <= 1/2
//   (Lanczos: x^5 ~ 5/4 h^2 x^3 - 5/16 h^4 x on |x| <= h, error h^5 / 16), which
//   leaves h^5 / 1920 = 1.4e-16 for h = pi / 1024; cos to f^4 (next term
//   1.2e-18).
// 12 FP64 operations; 256 entries with the series to rho^5 and rho^6 and a
// separate phase k r took 15.
constexpr int kFarTrigN = 1024;
constexpr double kFarTrigInvStep = 162.97466172610083;  // 1024 / (2 pi)
constexpr double kRoundMagic = 6755399441055744.0;      // 1.5 * 2^52
constexpr double kFarTrigStep = 0.006135923151542565;   // 2 pi / 1024
constexpr double kFarTrigH = 0.5 * kFarTrigStep;
constexpr double kFarS1 =
    kFarTrigStep * (1.0 - 5.0 / 16.0 / 120.0 * kFarTrigH * kFarTrigH * kFarTrigH * kFarTrigH);
constexpr double kFarS3 = kFarTrigStep * kFarTrigStep * kFarTrigStep *
                          (-1.0 / 6.0 + 5.0 / 4.0 / 120.0 * kFarTrigH * kFarTrigH);
constexpr double kFarC2 = -0.5 * kFarTrigStep * kFarTrigStep;
constexpr double kFarC4 = kFarTrigStep * kFarTrigStep * kFarTrigStep * kFarTrigStep / 24.0;

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

// sin and cos of k r, kstep = k N / (2 pi).
__device__ __forceinline__ void sincos_far(double r, double kstep, const double2* tab, double& s,
                                           double& c) {
  const double u = fma(r, kstep, kRoundMagic);
  const int j = __double2loint(u) & (kFarTrigN - 1);
  const double f = fma(r, kstep, kRoundMagic - u);
  const double f2 = f * f;
  const double sp = f * fma(f2, kFarS3, kFarS1);
  const double cp = fma(f2, fma(f2, kFarC4, kFarC2), 1.0);
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
