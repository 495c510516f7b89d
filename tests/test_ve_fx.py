"""The local solve in fixed point (csrc/ve_fx.cuh): on the CPU against the root in extended precision, on the GPU
against the FP64 iteration of the same call.

CPU tolerance: each law's argument is a Q9.54 number from three truncated products (4 units of 2^-54), which moves its
term by as much and the root by no more; 2^-51 leaves a factor of two.
"""
import ctypes
import subprocess

import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W

LD = np.longdouble


def cases(n, seed):
    """Residuals 1 - a s - sum exp(n_k ln s + c_k) with a known root: a random root, random shares of the terms."""
    rng = np.random.default_rng(seed)
    s = 2.0 ** rng.uniform(-3.9, 0.95, n)
    nk = np.exp(rng.uniform(np.log(0.3), np.log(127.0), (3, n)))
    nk[0, ::3] = 3.5
    nl = rng.integers(0, 8, n).astype(np.int32)
    g = rng.dirichlet([0.3] * 4, n).T ** rng.choice([1, 3, 9], n)
    g[1:][(nl >> np.arange(3)[:, None] & 1) == 0] = 0.0
    g[0] = np.where((g[0] == 0) | (nl == 0), 1.0, g[0])
    g[0, (nl > 0) & (rng.random(n) < 0.2)] = 0.0  # no linear term
    g /= np.maximum(g.sum(axis=0), 1e-30)
    with np.errstate(divide="ignore"):
        c = np.where(g[1:] > 0, np.log(np.maximum(g[1:], 1e-60)) - nk * np.log(s), 0.0)
    a = g[0] / s
    near = rng.uniform(-1, 1, n) * 2.0 ** -rng.uniform(16, 30, n) / np.where(nl > 0, nk.max(axis=0), 1.0)
    return nl, a, nk, c, (s * (1 + near)).astype(np.float32)


def test_root_on_the_host(tmp_path):
    src = tmp_path / "v.cpp"
    src.write_text('#include "ve_fx.cuh"\nextern "C" void run(long n, const int *nl, const double *a, const double *nk, const '
                   "double *c, const float *s0, int *ok, double *s, double *e) {\n  for (long i = 0; i < n; i++) {\n"
                   "    int64_t N[3], C[3]; float F[3]; mdz::VeFxRoot r;\n"
                   "    ok[i] = 0; bool in = true;\n"
                   "    for (int k = 0; k < 3; k++) {\n"
                   "      in = in && (!(nl[i] >> k & 1) || (c[k * n + i] < 149 && c[k * n + i] > -149));\n"
                   "      N[k] = mdz::fx_fixed<56>(mdz::fx_bits(nk[k * n + i])); F[k] = (float)nk[k * n + i];\n"
                   "      if (in) C[k] = mdz::fx_fixed<54>(mdz::fx_bits(c[k * n + i]));\n    }\n    if (!in) continue;\n"
                   "    ok[i] = mdz::ve_root_fx(nl[i], a[i], N, C, F, s0[i], r);\n    if (!ok[i]) continue;\n"
                   "    s[i] = mdz::fx_normalise(r.S, -62);\n"
                   "    for (int k = 0; k < 3; k++) e[k * n + i] = (nl[i] >> k & 1) ? mdz::fx_normalise(r.M[k], r.m[k] - 62) : 0.0;\n"
                   "  }\n}\n")
    lib = tmp_path / "v.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I", R.HERE + "/csrc", str(src),
                    "-o", str(lib)], check=True, capture_output=True)
    n = 200000
    nl, a, nk, c, s0 = cases(n, 3)
    ok, s, e = np.zeros(n, np.int32), np.zeros(n), np.zeros((3, n))
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_long] + [ctypes.c_void_p] * 8
    nk, c = np.ascontiguousarray(nk), np.ascontiguousarray(c)
    f(n, *[x.ctypes.data for x in (nl, a, nk, c, s0, ok, s, e)])
    inside = (np.abs(np.where(nl >> np.arange(3)[:, None] & 1, c, 0)) < 149).all(axis=0)
    assert ok[inside].mean() > 0.995  # what is near its root and in range is taken
    sel = ok == 1
    x, on = s0[sel].astype(LD), (nl[sel] >> np.arange(3)[:, None] & 1) == 1
    N, Cc, A = nk[:, sel].astype(LD), c[:, sel].astype(LD), a[sel].astype(LD)
    for _ in range(5):
        t = np.where(on, np.exp(N * np.log(x) + np.where(on, Cc, 0)), 0)
        x = x * (1 + (1 - A * x - t.sum(axis=0)) / (A * x + (N * t).sum(axis=0)))
    t = np.where(on, np.exp(N * np.log(x) + np.where(on, Cc, 0)), 0)
    es = np.abs((s[sel] - x) / x).astype(float)
    ee = np.where(on, np.abs(e[:, sel] - t) / np.where(on, t, 1), 0).astype(float) / np.maximum(N, 1).astype(float)
    print("root", es.max(), "terms over n", ee.max(), "taken", ok.mean())
    assert es.max() < 2.0 ** -51 and ee.max() < 2.0 ** -51


def material(kind):
    m = W.materials_plain_large(5)
    if kind == "high_n":  # exponents at and beyond the fixed-point range
        for p, n in enumerate((0.5, 20.0, 127.9, 128.0, 200.0)):
            m.pwlv[p], m.npwl[p] = 1, n
            m.Apwl[p] = 1e-14 / (1e8 ** n) if n < 30 else 1e-300
            m.pref_pwl[p] = 1.0 if n < 30 else 1e9 / (m.Apwl[p] ** (-1.0 / n))
            m.Qpwl[p], m.Vpwl[p], m.Fpwl[p] = 0.0, 0.0, 1.0
            m.linv[p] = m.expv[p] = 0
    if kind == "constant":
        for p in range(5):
            m.cstv[p], m.eta0[p] = 1, 10.0 ** (19 + p)
    if kind == "cold":  # laws hundreds of orders of magnitude apart
        for p in range(5):
            m.Qpwl[p] *= 4.0
    return m


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "high_n", "constant", "cold", "no_elastic", "hot", "typical"])
def test_gpu_fixed_against_fp64(kind):
    from golden.cases import _points, alloc_point_outputs
    rng = np.random.default_rng(7)
    n, m = 20000, material(kind)
    pin = _points(rng, n, 5, T=(1300.0, 3000.0) if kind == "hot" else (400.0, 1400.0), d=(1e-6, 1e-1))
    md = W.make_model(2, 2, 5)
    md.min_eta, md.max_eta = 1e5, 1e40
    if kind == "no_elastic":
        md.elastic = 0
        pin["C"][:] = 1e80  # no plastic return of a purely viscous stress
    got = []
    ctx = R.Context(0)
    for start in (R.DEFAULT_START, 0, 8):  # fixed point; the reference's start; FP32 steps and FP64 Newton
        ctx.set_warmstart(None, start)
        out = alloc_point_outputs(n)
        pi, po = R.make_points(pin, out)
        rc = ctx.points(md, m, pi, po, n)
        assert rc in (R.MDZ_OK, R.MDZ_EVE_ITER), rc
        got.append(out)
    ctx.close()
    fx, ref, fp64 = got
    assert (fx["status"] == fp64["status"]).all()
    fine = (ref["status"] == 0) & (fp64["status"] == 0)
    assert fine.mean() > 0.99
    assert (fx["iters"][fine] <= fp64["iters"][fine]).mean() > 0.999
    Eii = np.sqrt(0.5 * 2 * pin["Exx"] ** 2 + pin["Exz"] ** 2)
    for k in ("etaVE", "Txx", "Txz", "Eii_pwl", "Eii_exp", "Eii_lin", "Eii_cst"):
        # the iterations stop within 1e-13 Eii of the residual's root
        scale = np.maximum(np.abs(fp64[k]), Eii) if k.startswith("Eii") else np.abs(fp64[k])
        for other in (ref, fp64):
            err = np.abs(fx[k] - other[k])[fine] / np.maximum(scale[fine], 1e-300)
            assert err.max() < 1e-12, (kind, k, err.max(), int(err.argmax()))
