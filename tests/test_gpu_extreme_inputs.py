"""Inputs at the ends of what the calls accept, against the oracle: what is NaN there is NaN here, and errors are the same
errors."""
import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W
import oracle_lib as O
from common import clone
from golden.cases import alloc_point_outputs, point_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = R.Context(0)
    yield c
    c.close()


def run_points(ctx, name, change):
    md, m, pin, aniso, centroid, fu = point_case(name)
    n = pin["T"].size
    change(pin)
    out, ref = alloc_point_outputs(n), alloc_point_outputs(n)
    ctx.points(md, m, *R.make_points(pin, out, centroid=centroid, final_update=fu), n, aniso=int(aniso))
    O.orc_points(md, m, *R.make_points(pin, ref, centroid=centroid, final_update=fu), n, int(aniso))
    assert np.array_equal(out["status"], ref["status"])
    return out, ref


def run_sweeps(ctx, w, aniso=False):
    got, ref = clone(w.arrays), clone(w.arrays)
    rc, st = (ctx.sweep_aniso if aniso else ctx.sweep)(w.model, w.mat, R.FieldSet(got), check=False)
    orc, ost = O.orc_sweep(w.model, w.mat, R.FieldSet(ref), aniso=aniso)
    assert (rc, st.error_node) == (orc, ost.error_node)
    return got, ref


def same_nan(got, ref, fields):
    for k in fields:
        if ref.get(k) is not None:
            assert np.array_equal(np.isnan(got[k]), np.isnan(ref[k])), k


@pytest.mark.parametrize("name", ["popov", "gse", "constant_mix_gbs", "viscoplastic", "large_mix_peierls_cutoff"])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e300])
def test_points_with_a_strain_rate_that_is_not_finite(ctx, name, value):
    def change(pin):
        for k in ("Exx", "Exz"):
            pin[k][::3] = value
    out, ref = run_points(ctx, name, change)
    same_nan(out, ref, ["etaVE", "Txx", "Tzz", "Txz", "Pcorr"])


def test_anisotropic_points_with_an_infinite_strain_rate(ctx):
    out, ref = run_points(ctx, "aniso_mix", lambda pin: pin["Exx"].__setitem__(slice(None, None, 3), np.inf))
    same_nan(out, ref, ["etaVE", "Txx", "Tzz", "Txz", "Pcorr"])


@pytest.mark.parametrize("avg", [0, 1, 2])
@pytest.mark.parametrize("field", ["exxd", "ezzd", "exz_n", "sxxd0", "sxz0_n", "exxd_s", "exz", "sxz0"])
def test_sweeps_with_a_strain_rate_that_is_not_finite(ctx, field, avg):
    w = W.plain_large(seed=3, ncx=24, eta_average=avg)
    w.arrays[field][::7] = np.nan
    got, ref = run_sweeps(ctx, w)
    same_nan(got, ref, ["eta_n", "eta_s", "sxxd", "szzd", "sxz_n", "sxxd_s", "sxz", "eII_pl", "eII_pwl", "eII_lin", "p_corr"])
    for s in "ns":
        same_nan(dict(enumerate(got["phase_eta_" + s])), dict(enumerate(ref["phase_eta_" + s])), range(5))


@pytest.mark.parametrize("value", [0.0, 1e-310, 1e-300, np.nan])
def test_sweeps_without_a_finite_bulk_modulus_over_a_step(ctx, value):
    """K dt is infinite: a yielding node's return has no pressure, and the harmonic average is an error."""
    for avg in (0, 1):
        w = W.plain_large(seed=3, ncx=24, eta_average=avg)
        for s in "ns":
            w.arrays["bet_" + s][::5] = value
        got, ref = run_sweeps(ctx, w)
        same_nan(got, ref, ["eta_n", "eta_s", "sxxd", "sxz_n", "sxxd_s", "p_corr"])


@pytest.mark.parametrize("low,high", [(1e18, 1e17), (1e18, 1e-5), (1e18, 0.0)])
def test_anisotropic_limits_that_cross(ctx, low, high):
    """The upper limit is applied last to the visco-elastic and the visco-plastic viscosity."""
    w = W.aniso(seed=3, ncx=24)
    w.model.min_eta, w.model.max_eta = low, high
    got, ref = run_sweeps(ctx, w, aniso=True)
    for k in ("eta_n", "eta_s"):
        assert np.allclose(got[k], ref[k], rtol=1e-12, atol=0.0, equal_nan=True), k


def test_sweep_with_a_negative_shear_modulus(ctx):
    """Stress and viscosity are negative, and the dissipation is not: no error."""
    w = W.plain_large(seed=3, ncx=24)
    w.arrays["mu_n"][::7] = -1.0
    run_sweeps(ctx, w)
