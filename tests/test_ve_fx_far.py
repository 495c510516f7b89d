"""The local solve in fixed point (csrc/ve_fx.cuh) declines a start far from the root, also where the residual's Q2.62 sum
wraps round to near zero: terms of up to 2 and 1.82 add up to 5 while the number holds [-2, 2)."""
import ctypes
import subprocess

import numpy as np

import mdz_rheo as R

SOURCE = r"""
#include "ve_fx.cuh"
using namespace mdz;
extern "C" void run(long n, const double *a, const double *nk, const double *c, const float *s0, int *root, int *near_) {
  for (long i = 0; i < n; i++) {
    int64_t N[3], C[3], R;
    float nf[3];
    for (int k = 0; k < 3; k++) {
      N[k] = fx_fixed<56>(fx_bits(nk[k * n + i])); C[k] = fx_fixed<54>(fx_bits(c[k * n + i])); nf[k] = (float)nk[k * n + i];
    }
    VeFxRoot r;
    root[i] = ve_root_fx(7, a[i], N, C, nf, s0[i], r);
    const bool in = ve_residual_fx(7, a[i], N, C, (double)s0[i], R);  // the operators' test, |r| < 7e-14
    near_[i] = in && R < 322818 && R > -322818;
  }
}
"""


def test_wrapped_residuals_are_declined(tmp_path):
    src, lib = tmp_path / "v.cpp", tmp_path / "v.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", R.HERE + "/csrc", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    rng = np.random.default_rng(11)
    n = 20000
    s0 = (2.0 ** rng.uniform(-3.9, 0.95, n)).astype(np.float32)
    s = s0.astype(np.float64)
    nk = np.exp(rng.uniform(np.log(0.3), np.log(20.0), (3, n)))
    E = rng.uniform(1.02, 1.8, (3, n))
    lin = 5.0 - E.sum(axis=0)  # a s: the residual is 1 - 5, zero modulo 4
    keep = (lin > 0.05) & (lin < 1.99)
    c = np.log(E) - nk * np.log(s)
    a = lin / s
    root, near = np.ones(n, np.int32), np.ones(n, np.int32)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_long] + [ctypes.c_void_p] * 6
    f(n, *[x.ctypes.data for x in (a, nk, c, s0, root, near)])
    assert keep.sum() > 1000
    assert not root[keep].any() and not near[keep].any()
