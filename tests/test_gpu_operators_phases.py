"""The Newton operator with more phases than it keeps the strain-rate-independent part of the laws for: its compacting form
against the form with one thread per node, which keeps none, bit for bit."""
import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W
from common import clone

pytestmark = pytest.mark.gpu
OPS_PER_NODE = 0x40


@pytest.mark.parametrize("nphases", [1, 5, 6, 7, 8, 12, 20])
def test_phase_counts(nphases):
    mat = W.materials_plain_large(nphases, phase_ids=[k % 5 for k in range(nphases)])
    for p in range(nphases):  # no two phases alike
        mat.Apwl[p] *= 1.0 + 0.1 * p
    w = W.grid_workload("phases", 41, 37, mat, 5, grain_size=(1e-5, 1e-2), softening=(30.0, 5.0, 0.0, 1.0))
    a = clone(w.arrays)
    ctx = R.Context(0)
    try:
        ctx.sweep(w.model, mat, R.FieldSet(a))
        out = []
        for flags in (0, OPS_PER_NODE):
            o = R.alloc_operator_fields(w.Nc, w.Nv)
            assert ctx.operators(w.model, mat, R.FieldSet(a), o, flags=flags)[0] == R.MDZ_OK
            out.append(o)
    finally:
        ctx.close()
    for k in R.OPS_N + R.OPS_S:
        assert np.isfinite(out[0][k]).all() and np.array_equal(out[0][k], out[1][k]), k
