"""Sweeps and points whose plastic return is viscoplastic with a power law (n_vp != 1: the iterated return, with a power in
every pass) against the oracle, within the parity bar of the other sweeps."""
import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W
import oracle_lib as O
from common import RTOL, clone, worst
from golden.cases import _points, alloc_point_outputs

pytestmark = pytest.mark.gpu


def set_law(mat, eta_vp, n_vp):
    for p in range(mat.Nb_phases):
        mat.eta_vp[p], mat.n_vp[p] = eta_vp, n_vp


@pytest.mark.parametrize("eta_vp,n_vp", [(1e12, 2.0), (1e15, 1.5)])
def test_sweep_matches_oracle(eta_vp, n_vp):
    w = W.plain_large(seed=3, ncx=49)
    set_law(w.mat, eta_vp, n_vp)
    ref, got = clone(w.arrays), clone(w.arrays)
    assert O.orc_sweep(w.model, w.mat, R.FieldSet(ref))[0] == R.MDZ_OK
    ctx = R.Context(0)
    try:
        rc, st = ctx.sweep(w.model, w.mat, R.FieldSet(got))
    finally:
        ctx.close()
    assert rc == R.MDZ_OK and st.plastic_calls > 1000
    errors = worst(got, ref, w.arrays, w.model)
    assert max(errors.values()) <= RTOL, errors


def test_points_match_oracle():
    n, m = 4000, W.materials_plain_large(5)
    set_law(m, 1e12, 2.0)
    md = W.make_model(2, 2, 5)
    pin = _points(np.random.default_rng(5), n, 5)
    out, ref = alloc_point_outputs(n), alloc_point_outputs(n)
    O.orc_points(md, m, *R.make_points(pin, ref), n)
    ctx = R.Context(0)
    try:
        assert ctx.points(md, m, *R.make_points(pin, out), n) == R.MDZ_OK
    finally:
        ctx.close()
    assert np.array_equal(out["status"], ref["status"])
    Eii = np.sqrt(pin["Exx"] ** 2 + pin["Exz"] ** 2)
    for k in ("etaVE", "Txx", "Txz", "Pcorr", "Eii_pl"):
        scale = np.maximum(np.abs(ref[k]), Eii) if k == "Eii_pl" else np.abs(ref[k])
        assert np.max(np.abs(out[k] - ref[k]) / np.maximum(scale, 1e-300)) <= 10 * RTOL, k
