"""A mesh spacing that is not positive puts every marker outside the grid: an error status, not stresses of some other
cell."""
import pytest

import mdz_rheo as R
import mdz_workloads as W
from common import clone

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sx,sz,status", [(1, 1, R.MDZ_OK), (-1, 1, R.MDZ_EMARKER_OUT), (1, -1, R.MDZ_EMARKER_OUT)])
def test_spacing(sx, sz, status):
    w = W.marker_workload(seed=23, ncx=20, ncz=17, markers_per_cell=4)
    o = R.MarkerOpts()
    o.elastic, o.stress_rotation, o.anisotropy, o.advection, o.interp_stencil = 1, 1, 0, 1, 1
    ctx = R.Context(0)
    try:
        rc, _ = ctx.marker_stress(w.model, o, clone(w.arrays), clone(w.info["markers"]), sx * w.info["dx"], sz * w.info["dz"],
                                  check=False)
    finally:
        ctx.close()
    assert rc == status
