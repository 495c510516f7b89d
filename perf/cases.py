"""Measured cases of the local rheology library: what a geodynamics run calls in every time step, through the
public entry points of mdz_rheo.py.

A time step of MDOODZ interpolates marker fields to the grid (P2Mastah), prepares strengths and moduli, then for
each non-linear iteration forms the strain rates, updates the rheology of every node (the sweep) and builds the
viscosity operators of the momentum equations, and finally carries the stresses back to the markers.  The cases are
these calls, on device-resident fields (a solver on the GPU) and on host arrays (the drop-in), from a few thousand
points to the 2049 x 2049 benchmark grid.  The learned warm start is left out: it is an option that the default
start beats on every workload here, and its training is done once per network.

`exact` restates each path in torch float64 without the library (converged local solves, closed-form returns).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("mdoodz7.0_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mdz_rheo as R  # noqa: E402
import mdz_workloads as W  # noqa: E402

F8 = torch.float64
_CTX = []


def _ctx():
    """The program's one library context, on a stream that torch's copies can be ordered with."""
    if not _CTX:
        c, s = R.Context(0), torch.cuda.Stream()
        c.set_stream(s.cuda_stream)
        _CTX.extend((c, s))
    return _CTX[0]


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # ViscosityConcise on a few thousand loose points (a tabulation, a 0-D test): launch and latency count
        dict(name="points_2k", kind="points", n=2000, nph=5, seed0=3),
        # the 201 x 201 cell, 2-phase grid of the small benchmark: an ordinary 2-D model of a desktop run
        dict(name="sweep_201", kind="sweep", nx=201, nz=201, nph=2, avg=0, air=0.0, periodic=0),
        # a ragged grid with a free surface, periodic sides and the harmonic phase average
        dict(name="sweep_air_517x389", kind="sweep", nx=517, nz=389, nph=4, avg=1, air=0.2, periodic=1),
        # the headline benchmark: 2049 x 2049 cells, 5 phases of mixed creep laws
        dict(name="sweep_2049", kind="sweep", nx=2049, nz=2049, nph=5, avg=0, air=0.0, periodic=0),
        # the drop-in: the same sweep on the simulation's ordinary malloc'd host arrays
        dict(name="sweep_host_1025x769", kind="sweep_host", nx=1025, nz=769, nph=5, avg=0, air=0.0, periodic=0),
        # the anisotropic sweep of the 3-phase benchmark at a production size
        dict(name="aniso_1025", kind="aniso", nx=1025, nz=1025, nph=3, avg=0, air=0.0, periodic=0),
        # 16 uneven grids swept together, a captured time step of 5 sweeps with perturbed strain rates
        dict(name="batch_16x5", kind="batch", n=16, lo=65, hi=513, sweeps=5, seed0=7),
        # the Newton operator: 8 perturbed local solves per node and phase
        dict(name="newton_513", kind="newton", nx=513, nz=513, nph=5, avg=0, air=0.0, periodic=0),
        # velocity to strain rates, before every sweep
        dict(name="strain_rates_1025", kind="strain", nx=1025, nz=1025, air=0.1, periodic=0),
        # strain softening and shear moduli of a grid, once per time step
        dict(name="prep_1025", kind="prep", nx=1025, nz=1025, nph=5, air=0.1, periodic=0),
        # the marker stress update, 16 markers per cell as MDOODZ seeds them
        dict(name="markers_513", kind="markers", nx=513, nz=513, mpc=16, stencil=1, rotation=1, director=0),
        # a marker field onto centroids and vertices with the 9-cell stencil and the harmonic average
        dict(name="p2mastah_513", kind="p2m", nx=513, nz=513, mpc=16, stencil=9, avg=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "sweep", "sweep", "sweep_host", "aniso", "batch", "newton", "strain", "prep",
                       "markers", "p2m"])
    air, per = rng.choice([0.0, 0.0, 0.15, 0.3]), rng.choice([0, 0, 1])
    if kind == "points":
        return dict(kind=kind, n=_log_int(rng, 500, 200000), nph=rng.randint(1, 5), seed0=rng.randint(1, 99))
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(4, 24), lo=33, hi=_log_int(rng, 129, 513), sweeps=rng.randint(2, 6),
                    seed0=rng.randint(1, 99))
    top = {"sweep": 1500, "sweep_host": 900, "aniso": 1300, "newton": 500, "strain": 2049, "prep": 2049,
           "markers": 600, "p2m": 500}[kind]
    low = {"sweep": 65, "newton": 65}.get(kind, 129)
    nx, nz = _log_int(rng, low, top), _log_int(rng, low, top)
    if kind == "strain":
        return dict(kind=kind, nx=nx, nz=nz, air=air, periodic=per)
    if kind == "prep":
        return dict(kind=kind, nx=nx, nz=nz, nph=rng.randint(2, 8), air=air, periodic=per)
    if kind == "markers":
        return dict(kind=kind, nx=nx, nz=nz, mpc=rng.choice([4, 9, 16]), stencil=rng.choice([1, 9]),
                    rotation=rng.choice([1, 2]), director=rng.choice([0, 1]))
    if kind == "p2m":
        return dict(kind=kind, nx=nx, nz=nz, mpc=rng.choice([4, 9, 16]), stencil=rng.choice([1, 9]),
                    avg=rng.choice([0, 1, 2]))
    nph = rng.randint(1, 3) if kind == "aniso" else rng.randint(1, 5)
    return dict(kind=kind, nx=nx, nz=nz, nph=nph, avg=0 if kind == "newton" else rng.choice([0, 0, 1, 2]),
                air=air, periodic=per)


# ---- inputs, made on the GPU with the distributions of mdz_workloads ---------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _u(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=F8)


def _logu(g, n, lo, hi):
    return torch.exp(_u(g, n, math.log(lo), math.log(hi)))


def _sign(g, n):
    return torch.where(torch.rand(n, generator=g, device="cuda") < 0.5, -1.0, 1.0).to(F8)


def _modes(rng, modes=6, kmax=3):
    return [(int(rng.integers(-kmax, kmax + 1)), int(rng.integers(-kmax, kmax + 1)), rng.uniform(0, 2 * np.pi),
             rng.normal()) for _ in range(modes)]


def _smooth(modes, xs, zs):
    """One smooth random field (low-wavenumber plane waves, unit variance) on the tensor grid zs x xs."""
    out = torch.zeros(zs.numel(), xs.numel(), dtype=F8, device="cuda")
    for kx, kz, ph, amp in modes:
        a, b = 2 * math.pi * kx * xs + ph, 2 * math.pi * kz * zs
        out += amp * (torch.outer(torch.cos(b), torch.cos(a)) - torch.outer(torch.sin(b), torch.sin(a)))
    sd = out.std()
    return out / sd if float(sd) > 0 else out


def _coords(nx, nz):
    ar = lambda n: torch.arange(n, device="cuda", dtype=F8)  # noqa: E731
    return (ar(nx) + 0.5) / nx, (ar(nz) + 0.5) / nz, ar(nx + 1) / nx, ar(nz + 1) / nz


def _fractions(rng, nph, xs, zs, sharp=3.0):
    f = torch.stack([_smooth(m, xs, zs) for m in rng])
    return torch.softmax(sharp * f, dim=0).reshape(nph, -1)


def _flags(nx, nz, air, phase):
    """BC flags of cells and vertices: air (30) above a wavy surface, 31 in the row of cells below it."""
    xc, zc, xv, zv = _coords(nx, nz)
    p = torch.full((nz, nx), -1, dtype=torch.int8, device="cuda")
    g = torch.full((nz + 1, nx + 1), -1, dtype=torch.int8, device="cuda")
    if air > 0:
        h = 1.0 - air + 0.05 * torch.sin(4 * math.pi * xc + phase)
        above = zc[:, None] > h[None, :]
        p[above] = 30
        p[(~above) & (zc[:, None] > h[None, :] - 1.0 / nz)] = 31
        hv = 1.0 - air + 0.05 * torch.sin(4 * math.pi * xv + phase)
        g[zv[:, None] > hv[None, :]] = 30
        r = torch.nn.functional.pad((p < 30), (1, 1, 1, 1))  # a vertex between air cells only is air too
        g[~(r[:-1, :-1] | r[:-1, 1:] | r[1:, :-1] | r[1:, 1:])] = 30
    return p.reshape(-1), g.reshape(-1)


def _grid_fields(nx, nz, mat, seed, aniso=False, air=0.0, grain=True, out=None):
    """Every array of a sweep on nx x nz cells: T ~ U(500, 1400) K, lithostatic P, log-uniform strain rates of
    either sign, old stresses +-50 MPa, softmax phase fractions, friction softened 30 to 5 degrees.  `out`: where
    to take the arrays from (a batch keeps each field of its grids in one tensor)."""
    g, rng = _gen(seed), np.random.default_rng(seed)
    nph, nc, nv = mat.Nb_phases, nx * nz, (nx + 1) * (nz + 1)
    xc, zc, xv, zv = _coords(nx, nz)
    modes = [_modes(rng) for _ in range(nph)]
    a = {}
    bp, bg = _flags(nx, nz, air, rng.uniform(0, 2 * math.pi))
    a["BCp_type"], a["BCg_type"] = bp, bg
    a["T"] = _u(g, nc, 500.0, 1400.0)
    a["T0_n"] = a["T"].clone()
    a["p_in"] = (3000.0 * 9.81 * 100e3 * (1.0 - zc)).repeat_interleave(nx)
    a["p0_n"] = a["p_in"].clone()
    a["p0_s"] = (3000.0 * 9.81 * 100e3 * (1.0 - zv)).repeat_interleave(nx + 1)
    a["d0_n"] = _logu(g, nc, 1e-5, 1e-2) if grain else torch.full((nc,), 2e-3, dtype=F8, device="cuda")
    for s, n, xs, zs in (("n", nc, xc, zc), ("s", nv, xv, zv)):
        a["phase_perc_" + s] = _fractions(modes, nph, xs, zs).contiguous()
        exx, exz = _logu(g, n, 1e-16, 1e-13) * _sign(g, n), _logu(g, n, 1e-16, 1e-13) * _sign(g, n)
        sxx, sxz = _u(g, n, -5e7, 5e7), _u(g, n, -5e7, 5e7)
        names = (("exxd", "ezzd", "exz_n", "sxxd0", "szzd0", "sxz0_n") if s == "n" else
                 ("exxd_s", "ezzd_s", "exz", "sxxd0_s", "szzd0_s", "sxz0"))
        for k, v in zip(names, (exx, -exx, exz, sxx, -sxx, sxz)):
            a[k] = v
        eps = _u(g, n, 0.0, 1.0)
        a["strain_" + s] = eps
        a["fric_" + s] = (30.0 - 25.0 * eps) * W.DEG
        for k, v in (("C_", 1e7), ("dil_", 0.0), ("mu_", 3e10), ("bet_", 1e-40), ("X0_", 0.0)):
            a[k + s] = torch.full((n,), v, dtype=F8, device="cuda")
        if aniso:
            th, fac = _u(g, n, 0.0, math.pi), _logu(g, n, 1.0, 10.0)
            c, s_ = torch.cos(th), torch.sin(th)
            a["d1_" + s], a["d2_" + s] = 2 * c ** 2 * s_ ** 2, c * s_ * (s_ ** 2 - c ** 2)
            a["angle_" + s], a["aniso_factor_" + s] = th, fac
    a["phi0_n"] = torch.zeros(nc, dtype=F8, device="cuda")
    a["div_u"] = torch.zeros(nc, dtype=F8, device="cuda")
    a["div_u_s"] = torch.zeros(nv, dtype=F8, device="cuda")
    for k in _outputs(aniso):
        n = nv if k in R.VER_INTERP + R.VER_OUT or k == "phase_eta_s" else nc
        shape = (nph, n) if k.startswith("phase_eta") else (n,)
        a[k] = torch.zeros(shape, dtype=F8, device="cuda")
    return a


def _outputs(aniso):
    return ([k for k in R.CEN_OUT if k != "rho_n"] + [k for k in R.VER_OUT if aniso or k != "VE_s"] + R.VER_INTERP
            + ["phase_eta_n", "phase_eta_s"])


def _fieldset(a):
    """The library's view of the arrays: phase tables as one contiguous row per phase."""
    return R.FieldSet({k: (list(v) if k.startswith("phase_") else v) for k, v in a.items()})


def _materials(nph, aniso=False):
    if not aniso:
        return W.materials_plain_small() if nph == 2 else W.materials_plain_large(nph)
    m = W.empty_materials(nph)
    for p in range(nph):
        W.set_power_law(m, p, **(W.OLIVINE_DRY, W.SOFT_QTZ, W.OLIVINE_DRY)[p % 3])
    return m


def _model(c, nph):
    md = W.make_model(c["nx"], c["nz"], nph, eta_average=c.get("avg", 0))
    md.periodic_x = c.get("periodic", 0)
    return md


def _point_inputs(n, nph, seed):
    g = _gen(seed)
    p = {"phase": torch.randint(0, nph, (n,), generator=g, device="cuda", dtype=torch.int32)}
    full = lambda v: torch.full((n,), v, dtype=F8, device="cuda")  # noqa: E731
    exx, txx = _logu(g, n, 1e-15, 1e-13) * _sign(g, n), _u(g, n, -5e7, 5e7)
    p.update(G=full(3e10), T=_u(g, n, 600.0, 1300.0), P=_u(g, n, 0.0, 3e9), d=_logu(g, n, 1e-4, 5e-3), phi=full(0.0),
             X0=full(0.0), Exx=exx, Ezz=-exx, Exz=_logu(g, n, 1e-15, 1e-13) * _sign(g, n), Txx0=txx, Tzz0=-txx,
             Txz0=_u(g, n, -5e7, 5e7), strain_acc=full(0.0), dil=full(0.0), fric=full(30.0 * W.DEG), C=full(1e7),
             beta=full(1e-40), div=full(0.0))
    p["P0"], p["T0"] = p["P"].clone(), p["T"].clone()
    return p


def _batch_grids(case, seed):
    """Uneven grids of the many-grid workload: log-uniform sides, 2 to 5 of the five phases each, dt 1e10-1e12 s.
    The shapes come from the case, the fields from the seed."""
    rng = np.random.default_rng(case["seed0"])
    out = []
    for k in range(case["n"]):
        side = int(round(float(W.loguniform(rng, case["lo"], case["hi"], 1)[0])))
        nph = int(rng.integers(2, 6))
        ids = sorted(rng.choice(5, size=nph, replace=False).tolist())
        dt = float(W.loguniform(rng, 1e10, 1e12, 1)[0])
        out.append((side, W.make_model(side, side, nph, dt=dt), W.materials_plain_large(nph, phase_ids=ids),
                    int(seed) * 1009 + k))
    return out


_RATES = ("exxd", "ezzd", "exz_n", "exxd_s", "ezzd_s", "exz")
_L = 1e5


def _velocity(nx, nz, seed):
    g, rng = _gen(seed), np.random.default_rng(seed)
    ar = lambda n, s: torch.arange(n, device="cuda", dtype=F8) + s  # noqa: E731
    out = []
    for xs, zs in ((ar(nx + 1, 0.0) / nx, ar(nz + 2, -0.5) / nz), (ar(nx + 2, -0.5) / nx, ar(nz + 1, 0.0) / nz)):
        f = _smooth(_modes(rng), xs, zs)
        out.append((1e-9 * (f + 0.01 * torch.randn(f.shape, generator=g, device="cuda", dtype=F8))).reshape(-1))
    return out


def _running(x0, step, n):
    return torch.from_numpy(np.concatenate([[x0], np.full(n - 1, step)]).cumsum()).cuda()


def _marker_state(c, seed):
    """Grid and markers of the stress update: markers uniform within each cell and stored cell by cell, 2 % of them
    inactive, stresses of 10 MPa with grid increments of 1 %."""
    nx, nz, mpc = c["nx"], c["nz"], c["mpc"]
    g, rng = _gen(seed), np.random.default_rng(seed)
    nc, nv = nx * nz, (nx + 1) * (nz + 1)
    dx, dz, x0, z0 = _L / nx, _L / nz, -0.5 * _L, -_L
    rn = lambda n: torch.randn(n, generator=g, device="cuda", dtype=F8)  # noqa: E731
    a = {"xg_coord": _running(x0, dx, nx + 1), "zg_coord": _running(z0, dz, nz + 1),
         "xvz_coord": _running(x0 - dx / 2, dx, nx + 2), "zvx_coord": _running(z0 - dz / 2, dz, nz + 2),
         "xc_coord": _running(x0 + dx / 2, dx, nx), "zc_coord": _running(z0 + dz / 2, dz, nz)}
    for k, n in (("sxxd", nc), ("szzd", nc), ("sxz", nv)):
        a[k] = 1e7 * rn(n)
        a[k + "0"] = a[k] * (1.0 + 0.01 * rn(n))
    a["u_in"], a["v_in"] = _velocity(nx, nz, seed + 1)
    a["wxz"] = 1e-14 * rn(nv)
    a["BCp_type"], a["BCg_type"] = _flags(nx, nz, 0.1, rng.uniform(0, 2 * math.pi))
    n = nc * mpc
    cell = torch.arange(nc, device="cuda").repeat_interleave(mpc)
    m = {"x": x0 + ((cell % nx) + torch.rand(n, generator=g, device="cuda", dtype=F8)) * dx,
         "z": z0 + ((cell // nx) + torch.rand(n, generator=g, device="cuda", dtype=F8)) * dz}
    ph = torch.randint(0, 3, (n,), generator=g, device="cuda", dtype=torch.int32)
    ph[torch.rand(n, generator=g, device="cuda") < 0.02] = -1
    th = _u(g, n, 0.0, 2 * math.pi)
    m.update(phase=ph, sxxd=1e7 * rn(n), szzd=1e7 * rn(n), sxz=1e7 * rn(n), nx=torch.cos(th), nz=torch.sin(th))
    return a, m, dx, dz


def prepare(case, seed):
    k = case["kind"]
    st = {"kind": k, "ctx": _ctx()}
    if k == "points":
        n, m = case["n"], W.materials_plain_large(case["nph"])
        pin = _point_inputs(n, case["nph"], seed)
        out = {q: torch.zeros(n, dtype=F8, device="cuda") for q in R.PT_OUT}
        out["status"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        md = W.make_model(2, 2, case["nph"])
        st.update(n=n, model=md, mat=m, keep=pin, out=out, structs=R.make_points(pin, out))
    elif k in ("sweep", "sweep_host", "aniso", "newton"):
        ani = k == "aniso"
        st["mat"], st["model"] = _materials(case["nph"], ani), _model(case, case["nph"])
        a = _grid_fields(case["nx"], case["nz"], st["mat"], seed, aniso=ani, air=case["air"],
                         grain=not ani and case["nph"] != 2)
        if k == "sweep_host":
            a = {q: v.cpu().numpy() for q, v in a.items()}
        st["fs"], st["out"] = _fieldset(a), {q: a[q] for q in _outputs(ani)}
        if k == "newton":  # the operator works on a grid that a sweep has just updated
            st["ctx"].sweep(st["model"], st["mat"], st["fs"], mem=R.MEM_DEVICE)
            nc, nv = case["nx"] * case["nz"], (case["nx"] + 1) * (case["nz"] + 1)
            ops = R.alloc_operator_fields(nc, nv, like=a["T"])
            ops["drhodp_n"] = None  # incompressible: the density derivative is not asked for
            st["ops"] = ops
        st["arrays"] = a
    elif k == "batch":
        grids = _batch_grids(case, seed)
        per = [_grid_fields(s, s, m, sd) for s, _, m, sd in grids]
        names = [q for q in per[0] if not q.startswith("phase_")]
        flat = {q: torch.cat([a[q] for a in per]) for q in names}
        for q in ("phase_perc_n", "phase_perc_s", "phase_eta_n", "phase_eta_s"):
            flat[q] = torch.cat([a[q].reshape(-1) for a in per])
        at, fss = {q: 0 for q in flat}, []
        for a in per:
            view = {}
            for q in flat:
                n = a[q].numel()
                view[q] = flat[q][at[q]:at[q] + n].view(a[q].shape)
                at[q] += n
            fss.append(_fieldset(view))
        st["saved"] = {q: flat[q].clone() for q in _RATES}
        b = R.Batch(st["ctx"], [md for _, md, _, _ in grids], [m for _, _, m, _ in grids], fss)
        b.capture(case["sweeps"], amp=0.05, seed=2026)
        st.update(batch=b, flat=flat, out={q: flat[q] for q in _outputs(False) + list(_RATES)})
    elif k == "strain":
        nc, nv = case["nx"] * case["nz"], (case["nx"] + 1) * (case["nz"] + 1)
        u, v = _velocity(case["nx"], case["nz"], seed)
        bp, bg = _flags(case["nx"], case["nz"], case["air"], float(np.random.default_rng(seed).uniform(0, 6.28)))
        sr = {"u_in": u, "v_in": v, "BCp_type": bp, "BCg_type": bg, **R.alloc_strain_rate_fields(nc, nv, like=u)}
        st.update(model=_model(case, 1), sr=sr, dx=_L / case["nx"], dz=_L / case["nz"],
                  out={q: sr[q] for q in R.SR_N + R.SR_S})
    elif k == "prep":
        nph = case["nph"]
        pm, a = _prep_inputs(case, seed)
        for q in R.SOFT_N + R.MOD_N:
            a[q] = torch.zeros(case["nx"] * case["nz"], dtype=F8, device="cuda")
        for q in R.SOFT_S + R.MOD_S:
            a[q] = torch.zeros((case["nx"] + 1) * (case["nz"] + 1), dtype=F8, device="cuda")
        fs = R.PrepFieldSet({q: (list(v) if q.startswith("phase_") else v) for q, v in a.items()})
        st.update(model=_model(case, nph), pm=pm, fs=fs, keep=a,
                  out={q: a[q] for q in R.SOFT_N + R.MOD_N + R.SOFT_S + R.MOD_S})
    else:
        a, m, dx, dz = _marker_state(case, seed)
        st.update(model=_model(case, 3), grid=a, markers=m, dx=dx, dz=dz)
        if k == "markers":
            o = R.MarkerOpts()
            o.elastic, o.stress_rotation, o.anisotropy, o.advection = 1, case["rotation"], case["director"], 1
            o.interp_stencil = case["stencil"]
            o.set_G([3e10, 2.5e10, 4e10])
            st["opts"] = o
            st["out"] = {q: m[q] for q in ("sxxd", "szzd", "sxz", "nx", "nz")} | {"wxz": a["wxz"]}
        else:
            st["values"] = _logu(_gen(seed + 5), m["x"].numel(), 1e-3, 1e-1)
            st["out"] = {"node_n": torch.zeros(case["nx"] * case["nz"], dtype=F8, device="cuda"),
                         "node_s": torch.zeros((case["nx"] + 1) * (case["nz"] + 1), dtype=F8, device="cuda")}
            st["args"] = (case["avg"], case["stencil"])
    torch.cuda.synchronize()
    return st


def _prep_inputs(case, seed):
    """Phase fractions with exact zeros (as marker interpolation leaves them), plastic strain in [0, 1.5), noise."""
    nx, nz, nph = case["nx"], case["nz"], case["nph"]
    g, rng = _gen(seed), np.random.default_rng(seed)
    pm = W.prep_materials(rng, nph)
    xc, zc, xv, zv = _coords(nx, nz)
    modes = [_modes(rng) for _ in range(nph)]
    sm = _modes(rng)
    a = {}
    for s, xs, zs in (("n", xc, zc), ("s", xv, zv)):
        f = _fractions(modes, nph, xs, zs)
        f = torch.where(f < 0.03, torch.zeros_like(f), f)
        a["phase_perc_" + s] = (f / f.sum(dim=0, keepdim=True)).contiguous()
        a["strain_pl_" + s] = (1.5 / (1.0 + torch.exp(-2.0 * _smooth(sm, xs, zs)))).reshape(-1)
        a["noise_" + s] = _u(g, xs.numel() * zs.numel(), -0.1, 0.1)
    a["BCp_type"], a["BCg_type"] = _flags(nx, nz, case["air"], float(rng.uniform(0, 6.28)))
    return pm, a


def run(st):
    k, ctx = st["kind"], st["ctx"]
    if k == "points":
        rc = ctx.points(st["model"], st["mat"], *st["structs"], st["n"], mem=R.MEM_DEVICE)
        if rc != R.MDZ_OK:
            raise R.RheoError(rc, "points")
    elif k == "sweep":
        ctx.sweep(st["model"], st["mat"], st["fs"], mem=R.MEM_DEVICE)
    elif k == "sweep_host":
        ctx.sweep(st["model"], st["mat"], st["fs"])
    elif k == "aniso":
        ctx.sweep_aniso(st["model"], st["mat"], st["fs"], mem=R.MEM_DEVICE)
    elif k == "newton":
        ctx.operators(st["model"], st["mat"], st["fs"], st["ops"], mem=R.MEM_DEVICE)
        return {q: v for q, v in st["ops"].items() if v is not None}
    elif k == "batch":
        with torch.cuda.stream(_CTX[1]):  # a launch is one time step: it starts from the step's strain rates
            for q, v in st["saved"].items():
                st["flat"][q].copy_(v)
        st["batch"].launch()
    elif k == "strain":
        ctx.strain_rates(st["model"], st["dx"], st["dz"], st["sr"], compressible=1.0, mem=R.MEM_DEVICE)
    elif k == "prep":
        ctx.softening(st["model"], st["pm"], st["fs"], marker_noise=1, mem=R.MEM_DEVICE)
        ctx.shear_modulus(st["model"], st["pm"], st["fs"], mem=R.MEM_DEVICE)
    elif k == "markers":
        ctx.marker_stress(st["model"], st["opts"], st["grid"], st["markers"], st["dx"], st["dz"], mem=R.MEM_DEVICE)
    else:
        o = st["out"]
        ctx.p2mastah(st["model"], st["grid"], st["markers"], st["values"], *st["args"], o["node_n"], o["node_s"],
                     st["dx"], st["dz"], mem=R.MEM_DEVICE)
    return st["out"]


# ---- what a pass cannot do without -------------------------------------------------------------------------------
# FP64 operations of one local solve as the reference states it: its creep laws (an exponential each), one evaluation
# of the converged residual (a power per law) and the post-processing, each exp or pow counted as 20
_SOLVE = 150


def work(case):
    k = case["kind"]
    if k == "points":
        return {"bytes": case["n"] * (8 * (19 + 24) + 8), "flops": case["n"] * _SOLVE}
    if k == "batch":
        g = _batch_grids(case, 0)
        w = [_sweep_work(s, s, m.Nb_phases, False) for s, _, m, _ in g]
        return {q: case["sweeps"] * sum(x[q] for x in w) for q in ("bytes", "flops")}
    nc, nv = case["nx"] * case["nz"], (case["nx"] + 1) * (case["nz"] + 1)
    if k in ("sweep", "sweep_host", "aniso"):
        return _sweep_work(case["nx"], case["nz"], case["nph"], k == "aniso")
    if k == "newton":
        return {"bytes": nc * (8 * (17 + case["nph"] + 8) + 1) + nv * (8 * (16 + case["nph"] + 4) + 1),
                "flops": 8 * case["nph"] * (nc + nv) * _SOLVE // 2}
    if k == "strain":
        return {"bytes": 8 * ((case["nx"] + 1) * (case["nz"] + 2) * 2 + 5 * (nc + nv)) + nc + nv, "flops": 30 * (nc + nv)}
    if k == "prep":
        return {"bytes": (nc + nv) * (8 * case["nph"] + 1 + 40) + nc * 24 + nv * 16,
                "flops": (nc + nv) * (12 + 12 * case["nph"])}
    n = nc * case["mpc"]
    if k == "markers":
        d = case["director"]
        return {"bytes": n * (68 + 32 * d) + 33 * nc + 33 * nv + d * 16 * nv, "flops": n * (60 + 60 * d)}
    return {"bytes": n * 28 + 9 * nc + 9 * nv + 8 * (nc + nv), "flops": n * 2 * (8 + 3 * case["stencil"])}


def _sweep_work(nx, nz, nph, ani):
    nc, nv, e = nx * nz, (nx + 1) * (nz + 1), 4 if ani else 0
    return {"bytes": nc * (8 * (18 + e + 2 * nph + 23) + 1) + nv * (8 * (13 + e + 2 * nph + 10 + int(ani)) + 1),
            "flops": (nc + nv) * nph * _SOLVE}


# ---- the same paths in torch float64 -----------------------------------------------------------------------------
def _laws(m, p, Eii, T, P, d, model):
    """Isolated viscosity (logarithm) and stress exponent of each active creep law, and ln(d^(m/n)) of diffusion."""
    lnE, laws = torch.log(Eii), {}
    if m.pwlv[p]:
        n = m.npwl[p]
        lnB = (math.log(m.pref_pwl[p] * m.Fpwl[p]) - math.log(m.Apwl[p]) / n) + (m.Qpwl[p] + P * m.Vpwl[p]) / (
            m.R * n * T)
        laws["pwl"] = (lnB + (1.0 / n - 1.0) * lnE, n)
    if m.linv[p]:
        n = m.nlin[p]
        lnB = (math.log(m.Flin[p]) - math.log(m.Alin[p]) / n) + (m.Qlin[p] + P * m.Vlin[p]) / (m.R * n * T)
        laws["lin"] = (lnB + m.mlin[p] / n * torch.log(d) + (1.0 / n - 1.0) * lnE, n)
    if m.expv[p]:
        gam, S = m.Gexp[p], m.Sexp[p]
        ea = m.Qexp[p] / m.R
        nE = ea / T * 2.0 * gam * (1.0 - gam) + m.nexp[p]
        lnA = math.log(math.sqrt(3.0) / 2.0) + math.log(m.Eexp[p]) + m.nexp[p] * math.log(gam * S) - ea / T * (
            1.0 - gam) ** 2
        laws["exp"] = (math.log(gam * S / math.sqrt(3.0)) + (lnE - lnA) / nE - math.log(2.0) - lnE, nE)
    return laws


def _ve_solve(Eii, eta_el, laws):
    """ln(eta) of the visco-elastic local solve, by Newton on ln(eta) from the upper bound, and Eii of each law."""
    u = torch.log(eta_el)
    for l, _ in laws.values():
        u = torch.minimum(u, l)
    for _ in range(30):
        el = torch.exp(u) / eta_el
        t = {k: torch.exp(n * (u - l)) for k, (l, n) in laws.items()}
        f = 1.0 - el - sum(t.values())
        u = u + f / (el + sum(n * t[k] for k, (_, n) in laws.items()))
    eta = torch.exp(u)
    return eta, {k: Eii * torch.exp(n * (u - l)) for k, (l, n) in laws.items()}


def _iso_phase(m, p, q, model):
    """ViscosityConcise of phase p at the nodes q (a dict of arrays), elastic, Drucker-Prager without viscoplasticity."""
    dt = model.dt
    Exx, Ezz, Exz = q["Exx"], q["Ezz"], q["Exz"]
    Eii = torch.sqrt(0.5 * (Exx ** 2 + Ezz ** 2 + (Exx + Ezz) ** 2) + Exz ** 2)
    eta_el = q["G"] * dt
    laws = _laws(m, p, Eii, q["T"], q["P"], q["d"], model)
    eta, e = _ve_solve(Eii, eta_el, laws)
    Tii = 2.0 * eta * Eii
    Ty = q["C"] * torch.cos(q["fric"]) + q["P"] * torch.sin(q["fric"])
    Kdt = dt / q["beta"]
    pl = Tii - Ty > 1e-17
    gdot = torch.where(pl, (Tii - Ty) / (eta + Kdt * torch.sin(q["fric"]) * torch.sin(q["dil"])), torch.zeros_like(Tii))
    Pc = q["P"] + torch.where(pl, Kdt * torch.sin(q["dil"]) * gdot, torch.zeros_like(gdot))
    T2 = Tii - eta * gdot
    ve = torch.where(pl, T2 / (2.0 * Eii), eta)
    inv = torch.zeros_like(eta)
    for k, v in e.items():
        t = 2.0 * v / Tii
        if k == "lin" and m.mlin[p] != 0.0:
            t = t * torch.exp(m.mlin[p] / m.nlin[p] * (torch.log(q["d"]) - math.log(m.gs_ref[p])))
        inv = inv + t
    inv = inv + torch.where(pl, gdot / T2, torch.zeros_like(gdot))
    s = [2.0 * ve * x for x in (Exx, Ezz, Exz)]
    ex, ez, exz = [(x - q[t]) / (2.0 * eta_el) for x, t in zip(s, ("Txx0", "Tzz0", "Txz0"))]
    z = torch.zeros_like(eta)
    lim = lambda x: x.clamp(model.min_eta, model.max_eta)  # noqa: E731
    o = {"eta": lim(1.0 / inv), "etaVE": lim(ve), "Txx": s[0], "Tzz": s[1], "Txz": s[2],
         "Eii_el": torch.sqrt(0.5 * (ex ** 2 + ez ** 2 + (ex + ez) ** 2) + exz ** 2), "Eii_pl": 0.5 * gdot,
         "Eii_pwl": e.get("pwl", z), "Eii_exp": e.get("exp", z), "Eii_lin": e.get("lin", z), "Eii_gbs": z,
         "Eii_cst": z, "inv_d1": z + 1.0 / m.gs_ref[p], "d1": z + m.gs_ref[p], "X1": q["X0"], "OverS": z, "Pcorr": Pc,
         "div_el": -(Pc - q["P0"]) / Kdt, "div_pl": gdot * torch.sin(q["dil"]), "Wtot": T2 ** 2 / eta,
         "Wel": T2 ** 2 / eta_el, "Wdiss": T2 ** 2 * inv, "rho": z + m.rho[p], "div_r": z, "VEcoeff": z}
    return o


def _aniso_phase(m, p, q, model):
    """ViscosityConciseAniso of phase p, elastic, power-law creep."""
    dt = model.dt
    Exx, Ezz, Exz = q["Exx"], q["Ezz"], q["Exz"]
    c, s = torch.cos(q["angle"] - math.pi / 2), torch.sin(q["angle"] - math.pi / 2)
    lx2, lxlz = c * c, c * s
    nz2 = 1.0 - lx2
    rxx = lx2 * Exx + nz2 * Ezz + 2 * lxlz * Exz
    rzz = nz2 * Exx + lx2 * Ezz - 2 * lxlz * Exz
    rxz = -lxlz * Exx + lxlz * Ezz + (lx2 - nz2) * Exz
    Eii = torch.sqrt(0.5 * (rxx ** 2 + rzz ** 2 + (rxx + rzz) ** 2) + rxz ** 2)
    eta_el = q["G"] * dt
    eta, e = _ve_solve(Eii, eta_el, _laws(m, p, Eii, q["T"], q["P"], q["d"], model))
    Tii = 2.0 * eta * Eii
    lim = lambda x: x.clamp(model.min_eta, model.max_eta)  # noqa: E731
    inv = sum(2.0 * v / Tii for v in e.values())
    eta = lim(eta)
    Ty = q["C"] * torch.cos(q["fric"]) + q["P"] * torch.sin(q["fric"])
    pl = Tii - Ty > 1e-17
    K = torch.sin(q["dil"]) * dt / q["beta"]
    gdot = torch.where(pl, (Tii - Ty) / (eta + K * torch.sin(q["fric"])), torch.zeros_like(Tii))
    T2 = torch.where(pl, Tii - gdot * eta, Tii)
    Pc = q["P"] + torch.where(pl, K * gdot, torch.zeros_like(gdot))
    ve = torch.where(pl, T2 / (2 * Eii), eta)
    inv = inv + gdot / T2
    z = torch.zeros_like(eta)
    return {"eta": lim(1.0 / inv), "etaVE": lim(ve), "Eii_el": T2 ** 2 * 0.25 / eta_el ** 2, "Eii_pl": 0.5 * gdot,
            "Eii_pwl": e.get("pwl", z), "Eii_exp": z, "Eii_lin": z, "Eii_gbs": z, "Eii_cst": z, "inv_d1": 1.0 / q["d"],
            "X1": z, "OverS": z, "Pcorr": Pc, "div_el": -(Pc - q["P0"]) * q["beta"] / dt,
            "div_pl": gdot * torch.sin(q["dil"]), "Wtot": T2 ** 2 / eta, "Wel": T2 ** 2 / eta_el, "Wdiss": T2 ** 2 * inv}


def _ring(f, nx, nz, per, solid):
    """Centroid field to vertices: the mean of the four cells of the ghost-ringed field, air cells as zero."""
    v = torch.where(solid, f, torch.zeros_like(f)).view(nz, nx)
    cols = [nx - 1 if per else 0] + list(range(nx)) + [0 if per else nx - 1]
    v = v[:, cols]
    v = torch.cat([v[:1], v, v[-1:]])
    return (0.25 * (v[:-1, :-1] + v[:-1, 1:] + v[1:, :-1] + v[1:, 1:])).reshape(-1)


def _effective(a, s, model, aniso):
    n = ("exxd", "ezzd", "exz_n", "sxxd0", "szzd0", "sxz0_n") if s == "n" else (
        "exxd_s", "ezzd_s", "exz", "sxxd0_s", "szzd0_s", "sxz0")
    exx, ezz, exz, sx, sz, sxz = (a[k] for k in n)
    eta_e = a["mu_" + s] * model.dt
    if not aniso:
        return exx + sx / (2 * eta_e), ezz + sz / (2 * eta_e), exz + sxz / (2 * eta_e), sx, sz, sxz
    f, d1, d2 = 1.0 - 1.0 / a["aniso_factor_" + s], a["d1_" + s], a["d2_" + s]
    A, B, C, D = 2 - 2 * f * d1, 2 * f * d1, 2 * f * d2, 1 + 2 * f * (d1 - 0.5)
    # the inverse of [[A, B, -C], [B, A, C], [-C, C, D]] by its adjugate
    a11, a12, a13 = D * A - C * C, -C * C - D * B, B * C + C * A
    a33 = A * A - B * B
    det = A * a11 + B * a12 - C * a13
    i = 1.0 / (det * eta_e)
    return (exx + (a11 * sx + a12 * sz + a13 * sxz) * i, ezz + (a12 * sx + a11 * sz - a13 * sxz) * i,
            exz + 0.5 * (a13 * sx - a13 * sz + a33 * sxz) * i, sx, sz, sxz)


def _exact_sweep(a, m, model, aniso, nx, nz):
    out = {k: torch.zeros_like(a[k]) for k in _outputs(aniso)}
    solid_c, solid_v = (a["BCp_type"] != 30) & (a["BCp_type"] != 31), a["BCg_type"] != 30
    for k, src in (("T_s", "T"), ("P_s", "p_in"), ("d0_s", "d0_n"), ("phi0_s", "phi0_n")):
        out[k] = torch.where(solid_v, _ring(a[src], nx, nz, model.periodic_x, solid_c), torch.zeros_like(out[k]))
    names = {"eII_el": "Eii_el", "eII_pl": "Eii_pl", "eII_pwl": "Eii_pwl", "eII_exp": "Eii_exp", "eII_lin": "Eii_lin",
             "eII_gbs": "Eii_gbs", "eII_cst": "Eii_cst", "p_corr": "Pcorr", "div_u_el": "div_el", "div_u_pl": "div_pl",
             "Wtot": "Wtot", "Wel": "Wel", "Wdiss": "Wdiss", "OverS_n": "OverS", "d_n": "inv_d1"}
    for s, solid in (("n", solid_c), ("s", solid_v)):
        at = solid.nonzero().reshape(-1)
        Exx, Ezz, Exz, sx, sz, sxz = (v[at] for v in _effective(a, s, model, aniso))
        q = {"Exx": Exx, "Ezz": Ezz, "Exz": Exz, "Txx0": sx, "Tzz0": sz, "Txz0": sxz, "G": a["mu_" + s][at],
             "T": (a["T"] if s == "n" else out["T_s"])[at], "P": (a["p_in"] if s == "n" else out["P_s"])[at],
             "d": (a["d0_n"] if s == "n" else out["d0_s"])[at], "fric": a["fric_" + s][at], "C": a["C_" + s][at],
             "dil": a["dil_" + s][at], "beta": a["bet_" + s][at], "P0": a["p0_" + s][at], "X0": a["X0_" + s][at]}
        if aniso:
            q["angle"] = a["angle_" + s][at]
        acc = {}
        for p in range(m.Nb_phases):
            o = (_aniso_phase if aniso else _iso_phase)(m, p, q, model)
            w = a["phase_perc_" + s][p][at]
            w = torch.where(w.abs() > 1e-13, w, torch.zeros_like(w))
            out["phase_eta_" + s][p][at] = torch.where(w != 0, o["etaVE"], torch.zeros_like(w))
            f = {0: lambda x: x, 1: lambda x: 1.0 / x, 2: torch.log}[model.eta_average]
            t = {"eta": f(o["etaVE"]), "eta_phys": f(o["eta"]), "X": o["X1"], "VE": o["etaVE"] / (q["G"] * model.dt)}
            if s == "n":
                t.update({k: o[v] for k, v in names.items()})
            for k, v in t.items():
                acc[k] = acc.get(k, 0.0) + w * v
        b = {0: lambda x: x, 1: lambda x: 1.0 / x, 2: torch.exp}[model.eta_average]
        eta, phys = b(acc["eta"]), b(acc["eta_phys"])
        if aniso:
            f, d1, d2 = (1.0 - 1.0 / a["aniso_factor_" + s])[at], a["d1_" + s][at], a["d2_" + s][at]
            t = (2 * eta * (Exx * (1 - f * d1) + Ezz * f * d1 - 2 * Exz * f * d2),
                 2 * eta * (Ezz * (1 - f * d1) + Exx * f * d1 + 2 * Exz * f * d2),
                 2 * eta * (-Exx * f * d2 + Ezz * f * d2 + 2 * Exz * (f * (d1 - 0.5) + 0.5)))
            out["VE_" + s][at] = acc["VE"]
        else:
            t = (2 * eta * Exx, 2 * eta * Ezz, 2 * eta * Exz)
        for k, v in zip(("sxxd", "szzd", "sxz_n") if s == "n" else ("sxxd_s", "szzd_s", "sxz"), t):
            out[k][at] = v
        out["eta_" + s][at], out["eta_phys_" + s][at], out["X_" + s][at] = eta, phys, acc["X"]
        if s == "n":
            for k in names:
                out[k][at] = 1.0 / acc[k] if k == "d_n" else acc[k]
    return out


def _exact_newton(a, m, model, nx, nz):
    """The central differences of the Newton operator (incompressible, arithmetic average) on exact local solves."""
    sw = _exact_sweep(a, m, model, False, nx, nz)
    out = {}
    for s, solid in (("n", (a["BCp_type"] != 30) & (a["BCp_type"] != 31)), ("s", a["BCg_type"] != 30)):
        at = solid.nonzero().reshape(-1)
        Exx, Ezz, Exz, sx, sz, sxz = (v[at] for v in _effective(a, s, model, False))
        base = {"Exx": Exx, "Ezz": Ezz, "Exz": Exz, "Txx0": sx, "Tzz0": sz, "Txz0": sxz, "G": a["mu_" + s][at],
                "T": (a["T"] if s == "n" else sw["T_s"])[at], "P": (a["p_in"] if s == "n" else sw["P_s"])[at],
                "d": (a["d0_n"] if s == "n" else sw["d0_s"])[at], "fric": a["fric_" + s][at], "C": a["C_" + s][at],
                "dil": a["dil_" + s][at], "beta": a["bet_" + s][at], "P0": a["p0_" + s][at], "X0": a["X0_" + s][at]}
        tol = 1e-5 if s == "n" else 1e-7
        dE = []
        for k, den in (("Exx", 2.0), ("Ezz", 2.0), ("Exz", 4.0), ("P", 2.0)):
            h = tol * base[k].abs() + tol / 1e10
            d = torch.zeros_like(h)
            for p in range(m.Nb_phases):
                hi, lo = (_iso_phase(m, p, {**base, k: base[k] + sg * h}, model)["etaVE"] for sg in (1.0, -1.0))
                w = a["phase_perc_" + s][p][at]
                d += torch.where(w.abs() > 1e-13, w, torch.zeros_like(w)) * (hi - lo)
            dE.append(d / (den * h))
        eta, z = sw["eta_" + s][at], torch.zeros_like(dE[0])
        rows = ((("D11_n", "D12_n", "D13_n", "D14_n"), Exx, (2 * eta, z, z, z)),
                (("D21_n", "D22_n", "D23_n", "D24_n"), Ezz, (z, 2 * eta, z, z))) if s == "n" else (
            (("D31_s", "D32_s", "D33_s", "D34_s"), Exz, (z, z, eta, z)),)
        for names, E, own in rows:
            for k, o, d in zip(names, own, dE):
                out[k] = torch.zeros(solid.numel(), dtype=F8, device="cuda")
                out[k][at] = o + 2.0 * d * E
    return out


def _splitmix(z):
    z = z + np.uint64(0x9e3779b97f4a7c15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
    return z ^ (z >> np.uint64(31))


def _exact_batch(case, seed):
    outs = []
    for gi, (side, md, m, sd) in enumerate(_batch_grids(case, seed)):
        a = _grid_fields(side, side, m, sd)
        nc = side * side
        with np.errstate(over="ignore"):
            for sw in range(case["sweeps"]):
                key = _splitmix(_splitmix(np.uint64(2026) ^ np.uint64(sw)) ^ np.uint64(gi))
                for comp, (kn, ks) in enumerate((("exxd", "exxd_s"), ("ezzd", "ezzd_s"), ("exz_n", "exz"))):
                    for k, off in ((kn, 0), (ks, nc)):
                        node = np.arange(a[k].numel(), dtype=np.uint64) + np.uint64(off)
                        h = _splitmix(key ^ (node * np.uint64(3) + np.uint64(comp)))
                        u = (h >> np.uint64(11)).astype(np.float64) * 2.0 ** -52 - 1.0
                        a[k] = a[k] * torch.from_numpy(1.0 + 0.05 * u).cuda()
        o = _exact_sweep(a, m, md, False, side, side)
        o.update({k: a[k] for k in _RATES})
        outs.append(o)
    return {k: torch.cat([o[k].reshape(-1) for o in outs]) for k in outs[0]}


def _exact_strain(case, seed):
    nx, nz = case["nx"], case["nz"]
    u, v = _velocity(nx, nz, seed)
    bp, bg = _flags(nx, nz, case["air"], float(np.random.default_rng(seed).uniform(0, 6.28)))
    sc, sv = (bp != 30) & (bp != 31), (bg != 30).view(nz + 1, nx + 1)
    dx, dz = _L / nx, _L / nz
    u, v = u.view(nz + 2, nx + 1), v.view(nz + 1, nx + 2)
    z = torch.zeros(nz, nx, dtype=F8, device="cuda")
    s2 = sc.view(nz, nx)
    dudx, dvdz = (u[1:-1, 1:] - u[1:-1, :-1]) / dx, (v[1:, 1:-1] - v[:-1, 1:-1]) / dz
    div = dudx + dvdz
    o = {"div_u": torch.where(s2, div, z), "exxd": torch.where(s2, dudx - div / 3, z),
         "ezzd": torch.where(s2, dvdz - div / 3, z)}
    zv = torch.zeros(nz + 1, nx + 1, dtype=F8, device="cuda")
    dudz, dvdx = (u[1:] - u[:-1]) / dz, (v[:, 1:] - v[:, :-1]) / dx
    exz, wxz = torch.where(sv, 0.5 * (dudz + dvdx), zv), torch.where(sv, 0.5 * (dvdx - dudz), zv)
    quad = lambda f: 0.25 * (f[:-1, :-1] + f[:-1, 1:] + f[1:, :-1] + f[1:, 1:])  # noqa: E731
    o.update(exz=exz, wxz=wxz, exz_n=torch.where(s2, quad(exz), z), wxz_n=torch.where(s2, quad(wxz), z))
    for k, src in (("exxd_s", "exxd"), ("ezzd_s", "ezzd"), ("div_u_s", "div_u")):
        o[k] = torch.where(sv.reshape(-1), _ring(o[src].reshape(-1), nx, nz, case["periodic"], sc), zv.reshape(-1))
    return {k: x.reshape(-1) for k, x in o.items()}


def _exact_prep(case, seed):
    pm, a = _prep_inputs(case, seed)
    nx, nz, out = case["nx"], case["nz"], {}
    for s, solid in (("n", (a["BCp_type"] != 30) & (a["BCp_type"] != 31)), ("s", a["BCg_type"] != 30)):
        e, z = a["strain_pl_" + s], torch.zeros_like(a["strain_pl_" + s])
        sums = [z.clone() for _ in range(6)]
        for p in range(case["nph"]):
            w = a["phase_perc_" + s][p]
            for i, (x, end, on) in enumerate(((pm.phi[p], pm.phi_end[p], pm.phi_soft[p]),
                                              (pm.psi[p], pm.psi_end[p], pm.psi_soft[p]),
                                              (pm.C[p], pm.C_end[p], pm.coh_soft[p]))):
                t = x + (end - x) / (pm.pls_end[p] - pm.pls_start[p]) * e
                t = torch.where(e < pm.pls_start[p], torch.full_like(e, x), t)
                t = torch.where(e >= pm.pls_end[p], torch.full_like(e, end), t)
                sums[i] += w * (t if on else x)
            sums[3] += w / pm.G[p]
            sums[4] += w / pm.bet[p]
            sums[5] += w * pm.alp[p]
        sums[2] = sums[2] * (1.0 + a["noise_" + s])
        f = [torch.where(solid, x, z) for x in (sums[0], sums[1], sums[2], 1.0 / sums[3], 1.0 / sums[4], sums[5])]
        if s == "s" and case["periodic"]:
            for x in f[3:5]:
                x = x.view(nz + 1, nx + 1)
                x[:, 0] = x[:, -1] = 0.5 * (x[:, 0] + x[:, -1])
        for k, x in zip(("fric_", "dil_", "C_", "mu_", "bet_"), f):
            out[k + s] = x
        if s == "n":
            out["alp"] = f[5]
    return out


def _exact_markers(case, seed):
    """The grid's stress increments at the markers by bilinear weights (an air corner lends its weight to the corner
    across), without the director; the spin onto vertices with a marker near them is zero."""
    a, m, dx, dz = _marker_state(case, seed)
    nx, nz, on = case["nx"], case["nz"], m["phase"] != -1
    x, z = m["x"], m["z"]

    def cells(x0, z0):
        fx, fz = (x - x0) / dx, (z - z0) / dz
        j, i = torch.floor(fx), torch.floor(fz)
        return j.long(), i.long(), fx - j, fz - i

    air_c, air_v = (a["BCp_type"] == 30) | (a["BCp_type"] == 31), (a["BCg_type"] == 30) | (a["BCg_type"] == 31)
    out = {}
    for s, names, air, w, (x0, z0) in (("n", ("sxxd", "szzd"), air_c, nx, (a["xc_coord"][0], a["zc_coord"][0])),
                                       ("s", ("sxz",), air_v, nx + 1, (a["xg_coord"][0], a["zg_coord"][0]))):
        h = nz if s == "n" else nz + 1
        j, i, fx, fz = cells(x0, z0)
        col = lambda k: k.clamp(0, w - 1)  # noqa: E731
        row = lambda k: k.clamp(0, h - 1)  # noqa: E731
        c = [col(j) + row(i) * w, col(j + 1) + row(i) * w, col(j) + row(i + 1) * w, col(j + 1) + row(i + 1) * w]
        wt = [(1 - fx) * (1 - fz), fx * (1 - fz), (1 - fx) * fz, fx * fz]
        for k in names:
            inc = torch.where(air if s == "n" else a["BCg_type"] == 30, torch.zeros_like(a[k]), a[k] - a[k + "0"])
            t = sum(wt[q] * inc[torch.where(air[c[q]], c[q ^ 2], c[q])] for q in range(4))
            out[k] = m[k] + torch.where(on, t, torch.zeros_like(t))
    out["nx"], out["nz"] = (None, None) if case["director"] else (m["nx"], m["nz"])
    out["wxz"] = None
    return out


def _exact_p2m(case, seed):
    a, m, dx, dz = _marker_state(case, seed)
    v = _logu(_gen(seed + 5), m["x"].numel(), 1e-3, 1e-1)
    on = m["phase"] != -1
    x, z, v = m["x"][on], m["z"][on], v[on]
    v = (v, 1.0 / v, torch.log(v))[case["avg"]]
    out = {}
    for s, xs, zs, air in (("n", a["xc_coord"], a["zc_coord"], (a["BCp_type"] == 30) | (a["BCp_type"] == 31)),
                           ("s", a["xg_coord"], a["zg_coord"], (a["BCg_type"] == 30) | (a["BCg_type"] == 31))):
        w, h = xs.numel(), zs.numel()
        j = (torch.ceil((x - xs[0]) / dx + 0.5).long() - 1).clamp(0, w - 1)
        i = (torch.ceil((z - zs[0]) / dz + 0.5).long() - 1).clamp(0, h - 1)
        W0, W1 = torch.zeros(w * h, dtype=F8, device="cuda"), torch.zeros(w * h, dtype=F8, device="cuda")
        r = range(-1, 2) if case["stencil"] == 9 else range(1)
        lx, lz = (1.5 * dx, 1.5 * dz) if case["stencil"] == 9 else (dx / 2, dz / 2)
        for di in r:
            for dj in r:
                ok = (i + di >= 0) & (i + di < h) & (j + dj >= 0) & (j + dj < w)
                ii, jj = (i + di)[ok], (j + dj)[ok]
                wt = (1 - (xs[j[ok]] + dj * dx - x[ok]).abs() / lx) * (1 - (zs[i[ok]] + di * dz - z[ok]).abs() / lz)
                W0.index_add_(0, jj + ii * w, wt)
                W1.index_add_(0, jj + ii * w, wt * v[ok])
        t = W1 / W0
        t = (t, 1.0 / t, torch.exp(t))[case["avg"]]
        out["node_" + s] = torch.where(air | (W0.abs() < 1e-30), torch.zeros_like(t), t)
    return out


def exact(case, seed):
    k = case["kind"]
    if k == "points":
        m, q = W.materials_plain_large(case["nph"]), _point_inputs(case["n"], case["nph"], seed)
        md = W.make_model(2, 2, case["nph"])
        o = [_iso_phase(m, p, q, md) for p in range(case["nph"])]
        ph = q["phase"].long()[None]
        out = {f: torch.stack([x[f] for x in o]).gather(0, ph)[0] for f in R.PT_OUT}
        return {**out, "status": None}
    if k in ("sweep", "sweep_host", "aniso", "newton"):
        ani = k == "aniso"
        m, md = _materials(case["nph"], ani), _model(case, case["nph"])
        a = _grid_fields(case["nx"], case["nz"], m, seed, aniso=ani, air=case["air"],
                         grain=not ani and case["nph"] != 2)
        if k == "newton":
            return _exact_newton(a, m, md, case["nx"], case["nz"])
        return _exact_sweep(a, m, md, ani, case["nx"], case["nz"])
    return {"batch": _exact_batch, "strain": _exact_strain, "prep": _exact_prep, "markers": _exact_markers,
            "p2m": _exact_p2m}[k](case, seed)
