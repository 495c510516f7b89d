"""fx_pow (csrc/fx64.cuh), the power of the sweeps' iterated plastic return, against extended precision: compiled for the
host on the CPU, and on the GPU through mdz_rheo_fx_pair_selftest.

Bound: the logarithm is within 2^-56 absolute (tests/test_fx64.py) and keeps 64 bits, as its product with y does; exp adds
0.5 ulp of rounding and less than 0.05 of its own.  For |y| < 1, |y log x| < 64 that is 0.5 + 0.25 + 0.05 ulp at most, and
2 ulp elsewhere (CUDA's pow or the C library's).
"""
import ctypes
import subprocess

import numpy as np
import pytest

import mdz_rheo as R

LD = np.longdouble


def arguments():
    rng = np.random.default_rng(13)
    n = 200000
    x = np.concatenate([np.exp(rng.uniform(-60, 60, n)), np.exp(rng.uniform(-45, -20, n)), np.exp(rng.uniform(-300, 300, n)),
                        rng.uniform(0.5, 2.0, n), 2.0 ** rng.integers(-80, 80, n).astype(float)])
    y = np.concatenate([rng.uniform(-1, 1, n), 1.0 / rng.uniform(1.01, 8, n) - 1.0, rng.uniform(-8, 8, n),
                        rng.uniform(-1, 1, n), rng.choice([-0.5, -0.75, 0.25, 1.0, -1.0, 2.0 ** -40, 0.0], n)])
    odd = [0.0, 1.0, np.inf, np.nan, 5e-324, 1e308, -2.0, 1e-300]
    ox, oy = np.meshgrid(odd, [-0.5, 0.0, 1.0, -1.0, 300.0, np.inf, np.nan])
    return np.concatenate([x, ox.ravel()]), np.concatenate([y, oy.ravel()])


def check(x, y, got):
    with np.errstate(all="ignore"):
        ref = np.power(x.astype(LD), y.astype(LD))
        d = ref.astype(np.float64)
        plain = np.isfinite(d) & (np.abs(d) > 2.3e-308)
        same = (got == d) | (np.isnan(got) & np.isnan(d)) | (np.abs(got - d) <= 1e-322)
        assert same[~plain].all()
        ulp = (np.abs(got.astype(LD) - ref) / np.spacing(np.abs(d))).astype(float)
        arg = np.abs(y * np.log(x))
        fast = plain & (x > 0) & (np.abs(np.log(x)) > 0.13) & (np.abs(y) < 1) & (arg < 64)
    print("fast", ulp[fast].max(), "else", ulp[plain & ~fast].max())
    assert fast.sum() > 300000 and ulp[fast].max() <= 0.8 and ulp[plain & ~fast].max() <= 2.0


def test_host_build(tmp_path):
    src, lib = tmp_path / "p.cpp", tmp_path / "p.so"
    src.write_text('#include "fx64.cuh"\nextern "C" void run(const double *x, const double *y, long n, double *o) {\n'
                   "  for (long i = 0; i < n; i++) o[i] = mdz::fx_pow(x[i], y[i]);\n}\n")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", R.HERE + "/csrc", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    x, y = arguments()
    out = np.empty(x.size)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]
    f(x.ctypes.data, y.ctypes.data, x.size, out.ctypes.data)
    check(x, y, out)


@pytest.mark.gpu
def test_gpu():
    x, y = arguments()
    fixed, cuda = R.fx_pair_selftest(x, y)[:2]
    check(x, y, fixed)
    with np.errstate(all="ignore"):
        ref = np.power(x.astype(LD), y.astype(LD))
        ulp = np.abs(cuda.astype(LD) - ref) / np.spacing(np.abs(ref.astype(np.float64)))
    print("CUDA's pow", float(np.nanmax(np.where(np.isfinite(ulp), ulp, 0))))
