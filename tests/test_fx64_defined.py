"""The fixed-point functions and the local solve in fixed point run without undefined behaviour (signed overflow, shifts of
or beyond what the language allows), over their ranges and where a number leaves its format: compiled for the host with
the compiler's checks as traps."""
import subprocess

import mdz_rheo as R

MAIN = r"""
#include <math.h>
#include <random>
#include "ve_fx.cuh"
using namespace mdz;
static uint64_t sink;
static void keep(double x) { sink ^= fx_bits(x); }
static void functions(double x) {
  keep(fx_exp(x)); keep(fx_log(x)); keep(fx_recip(x)); keep(fx_sqrt(x));
  double s, c;
  fx_sincos(x, &s, &c);
  keep(s); keep(c); keep(fx_mul_rn(x, s)); keep(fx_mul_rn(x, x)); keep(fx_pow(fabs(x), 0.9 * s));
}
static void solves(std::mt19937_64 &g, bool far) {
  std::uniform_real_distribution<double> u(0.0, 1.0);
  const int nl = (int)(g() & 7);
  const double s = exp2(-4.0 + 5.0 * u(g));
  int64_t N[3], C[3];
  float nf[3];
  for (int k = 0; k < 3; k++) {
    const double n = exp(log(0.3) + u(g) * log(127.9 / 0.3));
    double c = (far ? 280.0 * u(g) - 140.0 : log(u(g) + 1e-3)) - n * log(s);
    c = c < -148.0 ? -148.0 : (c > 148.0 ? 148.0 : c);
    N[k] = fx_fixed<56>(fx_bits(n)); C[k] = fx_fixed<54>(fx_bits(c)); nf[k] = (float)n;
  }
  const double a = far ? exp2(40.0 * u(g) - 20.0) : u(g) / s;
  VeFxRoot r;
  keep((double)ve_root_fx(nl, a, N, C, nf, (float)s, r));
  int64_t res;
  keep((double)ve_residual_fx(nl, a, N, C, s, res));
}
int main() {
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  for (int i = 0; i < 400000; i++) {
    functions(499.9 * u(g)); functions(u(g)); functions(40.0 * u(g) - 20.0);
    functions(ldexp(1.0 + fabs(u(g)), (int)(990 * u(g))));
    const uint64_t b = g();
    double x;
    memcpy(&x, &b, 8);
    functions(x);
    solves(g, false); solves(g, true);
  }
  for (int k = -1100; k <= 1100; k++) keep(fx_k_ln2(k));
  for (double x : {0.0, -0.0, 1.0, 2.0, 0.5, 500.0, -500.0, 1e308, 5e-324, HUGE_VAL, -HUGE_VAL, (double)NAN}) functions(x);
  return sink == 42;
}
"""


def test_no_undefined_behaviour(tmp_path):
    src, exe = tmp_path / "u.cpp", tmp_path / "u"
    src.write_text(MAIN)
    build = ["g++", "-O1", "-g", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I", R.HERE + "/csrc",
             str(src), "-o", str(exe)]
    if subprocess.run(build, capture_output=True).returncode != 0:  # no runtime library for the reports
        build[5:6] = ["-fsanitize-undefined-trap-on-error"]
        subprocess.run(build, check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
