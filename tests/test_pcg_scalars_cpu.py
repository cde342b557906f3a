"""Rounding of the mixed PCG's scalars, which run in float-float arithmetic:
quotients by a number whose reciprocal is at hand, and the step length alpha of
the single-reduction form, compiled for the host from the kernels' own header
and compared with long double.  Their errors, largest and rms, are no larger
than with FP64 products and differences between float-float divisions; for the
step after a failed verification, which takes its sums in FP64, the bound is
that of its two divisions: 2^-46.5 (the division's 2^-46.8, taken up) for beta."""
import shutil
import subprocess

import pytest

SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <algorithm>
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
#include "pcg_scalars.cuh"
using namespace mfem_gpu;
typedef long double Q;
static Q q(df64 v) { return (Q)v.hi + (Q)v.lo; }
static double div64(double a, double b) { return (df64(a) / df64(b)).to_double(); }
struct Err {
  double mx = 0, sq = 0;
  long n = 0;
  void add(Q v, Q exact) {
    const double e = std::fabs((double)((v - exact) / exact));
    mx = std::max(mx, e);
    sq += e * e;
    ++n;
  }
  void put() const { std::printf("%.9e %.9e\n", mx, std::sqrt(sq / n)); }
};
int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> U(0, 1);
  auto draw = [&]() { return df64(std::exp2(30 * U(g) - 15) * (1 + U(g))); };
  {
    Err ref, now;
    for (int i = 0; i < 400000; ++i) {
      const df64 n = draw(), d = draw();
      ref.add(div64(n.to_double(), d.to_double()), q(n) / q(d));
      now.add(q(by_rcp(n, d, rcp_of(d))), q(n) / q(d));
    }
    ref.put();
    now.put();
  }
  for (double cancel : {1.5, 4.0, 30.0, 300.0}) {
    Err ref, now;
    for (int i = 0; i < 400000; ++i) {
      const df64 gp = draw(), gn = draw(), ap = draw();
      const Q x = q(gn) / q(gp) * q(gn) / q(ap);
      const df64 d((double)(x / (1 - 1 / (Q)(cancel * (0.7 + 0.6 * U(g)) + 0.4))));
      const Q exact = q(gn) / (q(d) - x);
      const double b = div64(gn.to_double(), gp.to_double());
      ref.add(div64(gn.to_double(), d.to_double() - div64(b * gn.to_double(), ap.to_double())), exact);
      df64 an, bn;
      cgf_steps(gn, d, gp, ap, rcp_of(gp), rcp_of(ap), &an, &bn);
      now.add(q(an), exact);
    }
    ref.put();
    now.put();
  }
  Err beta;
  for (int i = 0; i < 400000; ++i) {
    const df64 su = draw(), ps = draw();
    df64 an, bn;
    cgf_restart_steps(draw(), draw(), su, ps, &an, &bn);
    beta.add(q(bn), -q(su) / q(ps));
  }
  beta.put();
  // step lengths: the same float as the quotient, also beside the middle of two
  long differ = 0;
  for (int i = 0; i < 400000; ++i) {
    const df64 d = draw();
    const float f = draw().hi, up = std::nextafterf(f, 2 * f);
    const double mid = 0.5 * ((double)f + up) * (1 + (i % 41 - 20) * std::exp2(-47 + i % 7));
    const df64 n = i % 2 ? df64(mid) * d : draw();
    differ += to_step(by_rcp_step(n, d, df64(1.f) / d)) != to_step(by_rcp(n, d, rcp_of(d)));
  }
  std::printf("%ld 0\n", differ);
  // dens whose reciprocal leaves FP32's range are divided by
  for (double den : {1e-38, 1e-31, 1e31, 1e38}) {
    const df64 d(den), n = df64(3.0) * d;
    std::printf("%.9e 0\n", std::fabs((double)(q(by_rcp(n, d, rcp_of(d))) / 3 - 1)));
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_scalar_errors_are_those_of_fp64_products_between_divisions(tmp_path):
    import os
    root = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
    src, exe = tmp_path / "scalars.cpp", tmp_path / "scalars"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(root, "mfem_gb300", "csrc"),
                    "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    rows = [tuple(map(float, l.split())) for l in subprocess.run([str(exe)], check=True, capture_output=True,
                                                                text=True).stdout.split("\n") if l]
    for ref, now in zip(rows[0:10:2], rows[1:10:2]):
        assert now[0] <= ref[0] and now[1] <= ref[1], (ref, now)
    assert rows[10][0] <= 2.0 ** -46.5
    assert rows[11][0] == 0
    # (near the ends of the range the low parts are subnormal: FP32's accuracy)
    assert all(r[0] <= 2.0 ** -23 for r in rows[12:])
