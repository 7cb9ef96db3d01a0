"""Sine and cosine of the FP64 far-field kernels (no GPU): trig_table.cuh compiled
for the host against 80-bit values of the exact product k r.

Largest error: the phase carries the rounding of k r (2^-53 of it) and j times
the rounding of 2 pi / 1024 (computed here).  The table value (half a unit in
the last place of a number below 1 in each component: 0.8e-16 together) and
the two fused additions (half a unit each, their products with sin rho < 2^-8
times smaller) add at most 2.5e-16, the series nothing that counts.

Root mean square for phases below 1: four roundings (two table values, two
additions) of 3.2e-17 each or less (a unit of 2^-53 / sqrt(12)), that of k r,
3.2e-17, and the step's part of the phase, 2.2e-17: 7.5e-17, below 8e-17."""
import os
import subprocess

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#define __device__
#define __forceinline__ inline
struct double2 { double x, y; };
static inline double2 make_double2(double a, double b) { return {a, b}; }
static struct { unsigned x; } threadIdx{0}, blockDim{1};
static inline void __syncthreads() {}
static inline int __double2loint(double v) { long long q; std::memcpy(&q, &v, 8); return int(q & 0xffffffffll); }
static inline void sincospi(double x, double* s, double* c) {
  const long double p = 3.14159265358979323846264338327950288L;
  *s = double(sinl(p * x)), *c = double(cosl(p * x));
}
using std::fma;
#define asm(...) ((void)0)  // device instructions of the other functions there
#include "trig_table.cuh"
int main() {
  using namespace bie::dev;
  static double2 tab[kFarTrigN];
  fill_far_trig_table(tab);
  srand48(1);
  const long double step = 2 * 3.14159265358979323846264338327950288L / 1024;
  const double rel = 0x1p-53 + double(fabsl((kFarTrigStep - step) / step));
  double worst = 0, rms = 0;
  const double ks[] = {0.37, 1.0, 2.0, 5.0, 7.3, 17.0}, tops[] = {1e-3, 1.0, 20.0, 100.0, 400.0};
  for (double k : ks)
    for (double top : tops) {
      double sum = 0;
      for (int i = 0; i < 60000; ++i) {
        // a third of the phases beside the edges of the table's steps
        double x = top * drand48();
        if (i % 3 == 0) x = (std::floor(x * 1024 / 6.283185307179586) + 0.5 + 1e-9 * (drand48() - 0.5)) * 6.283185307179586 / 1024;
        const double r = x / k;
        const long double ph = (long double)k * r;
        double s, c;
        sincos_far(k * r, tab, s, c);
        const double e = double(hypotl(s - sinl(ph), c - cosl(ph)));
        const double bound = 2.5e-16 + rel * double(ph);
        if (e / bound > worst) worst = e / bound;
        sum += e * e;
      }
      if (top == 1.0) rms = std::fmax(rms, std::sqrt(sum / 60000));
    }
  std::printf("%.4f %.3e\n", worst, rms);
  return 0;
}
"""


def test_sincos_far(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src, exe = tmp_path / "trig.cpp", tmp_path / "trig"
    src.write_text(SRC)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-ffp-contract=off",
                    "-D_GNU_SOURCE", "-march=x86-64-v3", "-I",
                    os.path.join(root, "fmm3dbie_b200", "csrc", "cuda"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    worst, rms = float(out[0]), float(out[1])
    print(f"\nlargest error: {worst:.2f} of the bound; root mean square up to 1: {rms:.2e}")
    assert worst <= 1.0
    assert rms <= 8e-17
