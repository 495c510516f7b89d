"""The fixed-point elementary functions (csrc/fx64.cuh) against extended precision: compiled for the host on the CPU,
and on the GPU through mdz_rheo_fx_selftest.

Bounds: a result is rounded once to 53 bits (0.5 ulp) after an evaluation whose error is below 2^-56 of the leading
bit, 2^-58 for the reciprocal and the square root: 0.7 and 0.52 ulp; the argument of exp is cut to a multiple of 2^-54
and that of log leaves up to 2^-56 absolute, half an ulp of the smallest results, on top: 1.1 ulp.  Outside their
ranges the functions are the C library's or CUDA's (2 ulp).
"""
import ctypes
import subprocess

import numpy as np
import pytest

import mdz_rheo as R

LD = np.longdouble
NAMES = ("exp", "log", "recip", "sqrt", "sin", "cos")


def arguments():
    rng = np.random.default_rng(5)
    n = 200000
    x = np.concatenate([
        rng.uniform(-499.9, 499.9, n), rng.uniform(-40, 1, n), rng.uniform(0, 1.5, n),
        rng.choice([-1.0, 1.0], n) * 2.0 ** rng.uniform(-60, 2, n), np.exp(rng.uniform(-690, 690, n)),
        2.0 ** rng.integers(-990, 990, 2000).astype(float),
        [0.0, -0.0, 1.0, -1.0, 2.0, 0.5, 500.0, -500.0, 499.99999, 700.0, -700.0, -750.0, 800.0, 1.4999999, 1.5, 0.0625,
         np.nextafter(0.0625, 0), 1.1331484530668263, 0.8824969025845955, np.nextafter(1.0, 0), np.nextafter(1.0, 2),
         np.nextafter(2.0, 0), np.nextafter(4.0, 0), 5e-324, 1e-310, 1.7e308, np.inf, -np.inf, np.nan]])
    k = np.arange(1, 256) / 256.0  # table steps, and their neighbours
    return np.concatenate([x, k, np.nextafter(k, 0), np.nextafter(k, 2), 1 + k, 1 + np.nextafter(k, 0),
                           k * np.log(2.0), -k * np.log(2.0), np.nextafter(k * np.log(2.0), 9)])


def reference(x):
    with np.errstate(all="ignore"):
        v = x.astype(LD)
        return np.exp(v), np.log(v), LD(1) / v, np.sqrt(v), np.sin(v), np.cos(v)


def check(x, got):
    with np.errstate(all="ignore"):
        for name, g, r in zip(NAMES, got, reference(x)):
            d = r.astype(np.float64)
            odd = ~np.isfinite(d) | (d == 0) | (np.abs(d) < 2.3e-308)
            if name in ("sin", "cos"):
                odd |= np.abs(x) > 10
            same = (g == d) | (np.isnan(g) & np.isnan(d)) | (odd & np.isfinite(d) & (np.abs(g - d) <= 4e-308 + 1e-15 * np.abs(d)))
            assert same[odd].all(), (name, x[odd][~same[odd]], g[odd][~same[odd]])
            ulp = np.abs((g.astype(LD) - r) / np.spacing(np.abs(d)))[~odd].astype(float)
            a, xa = np.abs(d[~odd]), np.abs(x[~odd])
            fast = {"exp": xa < 500, "log": a >= 0.1251, "recip": (xa > 2.0 ** -999) & (xa < 2.0 ** 999),
                    "sqrt": (xa > 2.0 ** -999) & (xa < 2.0 ** 999)}.get(name, (xa >= 0.0625) & (xa < 1.5))
            bound = {"exp": 1.1, "log": 1.1, "recip": 0.52, "sqrt": 0.52}.get(name, 0.7)
            worst = ulp[fast].max(), ulp[~fast].max(initial=0)
            print(name, "fast", worst[0], "else", worst[1])
            assert worst[0] <= bound and worst[1] <= 2.0, (name, worst, x[~odd][fast][ulp[fast].argmax()])


def test_host_build(tmp_path):
    src = tmp_path / "fx.cpp"
    src.write_text('#include "fx64.cuh"\nextern "C" void run(const double *x, long n, double *o) {\n'
                   "  for (long i = 0; i < n; i++) {\n    o[i] = mdz::fx_exp(x[i]); o[n + i] = mdz::fx_log(x[i]);\n"
                   "    o[2 * n + i] = mdz::fx_recip(x[i]); o[3 * n + i] = mdz::fx_sqrt(x[i]);\n"
                   "    mdz::fx_sincos(x[i], &o[4 * n + i], &o[5 * n + i]);\n  }\n}\n")
    lib = tmp_path / "fx.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", R.HERE + "/csrc", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    x = arguments()
    out = np.empty((6, x.size))
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]
    f(x.ctypes.data, x.size, out.ctypes.data)
    check(x, out)


@pytest.mark.gpu
def test_gpu():
    x = arguments()
    check(x, R.fx_selftest(x))


def test_k_ln2_on_the_host(tmp_path):
    """k ln 2 for every k that a normalisation can have: the bits of the FP64 form it stands in for (a product and a
    fused multiply-add with ln 2 in two parts), here in exact rational arithmetic."""
    from fractions import Fraction
    src = tmp_path / "k.cpp"
    src.write_text('#include "fx64.cuh"\nextern "C" double k_ln2(int k) { return mdz::fx_k_ln2(k); }\n')
    lib = tmp_path / "k.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", R.HERE + "/csrc", str(src), "-o", str(lib)],
                   check=True, capture_output=True)
    f = ctypes.CDLL(str(lib)).k_ln2
    f.restype = ctypes.c_double
    hi, lo = float.fromhex("0x1.62e42fefa39efp-1"), float.fromhex("0x1.abc9e3b39803fp-56")
    for k in range(-1100, 1101):
        assert f(k) == float(Fraction(k) * Fraction(hi) + Fraction(k * lo)), k


def test_division_near_one_on_the_host(tmp_path):
    """div_near_one against IEEE division, bit for bit: every divisor within its range, numerators random and at the
    ends of a binade, zeros; what it declines is left to the division."""
    src = tmp_path / "d.cpp"
    text = open(R.HERE + "/csrc/fp64_div.cuh").read()
    at = text.index("FX_FN bool div_near_one")
    src.write_text('#include "fx64.cuh"\nnamespace mdz {\n' + text[at:text.index("\n}\n", at) + 3] + "}\n"
                   'extern "C" void run(long n, const double *a, const double *s, double *q, int *ok) {\n'
                   "  for (long i = 0; i < n; i++) ok[i] = mdz::div_near_one(a[i], s[i], q[i]);\n}\n")
    lib = tmp_path / "d.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", R.HERE + "/csrc", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    rng = np.random.default_rng(9)
    n = 2_000_000
    s = (np.int64(0x3ff0000000000000) + rng.integers(-34, 19, n)).view(np.float64)
    man = rng.integers(0, 1 << 52, n)
    man[::5] = rng.integers(0, 300, man[::5].size)
    man[1::5] = (1 << 52) - 1 - rng.integers(0, 300, man[1::5].size)
    bits = (rng.integers(0, 2, n) << 63) | (rng.integers(0, 2048, n) << 52) | man
    a = bits.astype(np.uint64).view(np.float64)
    a[::97] = 0.0
    a[1::97] = -0.0
    q, ok = np.zeros(n), np.zeros(n, np.int32)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_long] + [ctypes.c_void_p] * 4
    f(n, *[x.ctypes.data for x in (a, s, q, ok)])
    with np.errstate(all="ignore"):
        want = a / s
    t = ok == 1
    assert t.mean() > 0.5 and np.array_equal(q[t].view(np.uint64), want[t].view(np.uint64))


def test_product_on_the_host(tmp_path):
    """fx_mul_rn against the FP64 multiplication, bit for bit: random bit patterns (every exponent, special values),
    short significands (exact products and ties), products near the ends of the range."""
    src = tmp_path / "m.cpp"
    src.write_text('#include "fx64.cuh"\nextern "C" void run(long n, const double *a, const double *b, double *o) {\n'
                   "  for (long i = 0; i < n; i++) o[i] = mdz::fx_mul_rn(a[i], b[i]);\n}\n")
    lib = tmp_path / "m.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", R.HERE + "/csrc", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    rng = np.random.default_rng(21)
    n = 3_000_000
    x, y = (rng.integers(0, 1 << 64, n, dtype=np.uint64) for _ in range(2))
    x[::3] &= np.uint64(0xfffffffff0000000)
    y[::3] &= np.uint64(0xffffffffff000000)
    for v, lo in ((x, 900), (y, 1000)):  # exponents near 1, so that most products are normal
        v[1::2] = (v[1::2] & np.uint64(0x800fffffffffffff)) | ((np.uint64(lo) + v[1::2] % np.uint64(100)) << np.uint64(52))
    x[5::50] = np.uint64(0)
    y[6::50] = np.uint64(1 << 63)
    a, b = x.view(np.float64), y.view(np.float64)
    o = np.empty(n)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_long] + [ctypes.c_void_p] * 3
    f(n, a.ctypes.data, b.ctypes.data, o.ctypes.data)
    with np.errstate(all="ignore"):
        want = a * b
    same = (o.view(np.uint64) == want.view(np.uint64)) | (np.isnan(o) & np.isnan(want))
    assert same.all(), (a[~same][:3], b[~same][:3])
