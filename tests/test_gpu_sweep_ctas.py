"""The register cap that a sweep's size selects (5 or 7 CTAs per SM) changes no bit: grids on both
sides of each line against the 255-register kernel."""
import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W
from common import clone

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WAVE = 152 * 7 * 128


def to_device(arrays):
    return {k: ([torch.from_numpy(x).cuda() for x in v] if isinstance(v, list) else torch.from_numpy(v).cuda())
            for k, v in arrays.items()}


@pytest.mark.parametrize("aniso", [False, True])
@pytest.mark.parametrize("ncx,five", [(259, False), (262, True), (486, True), (489, False)])
def test_register_cap_keeps_the_bits(aniso, ncx, five):
    w = W.aniso(seed=3, ncx=ncx) if aniso else W.plain_large(seed=3, ncx=ncx)
    assert (WAVE < w.nodes and 2 * w.nodes < 7 * WAVE) == five
    ctx = R.Context(0)
    try:
        fn = ctx.sweep_aniso if aniso else ctx.sweep
        out = []
        for form in (0, 1):
            ctx.set_launch_shape(aniso, 128, 0, form)
            d = to_device(clone(w.arrays))
            torch.cuda.synchronize()
            fn(w.model, w.mat, R.FieldSet(d), mem=R.MEM_DEVICE)
            out.append(d)
        for k in R.CEN_OUT + R.VER_OUT:
            if out[0].get(k) is not None:
                assert np.array_equal(out[0][k].cpu().numpy(), out[1][k].cpu().numpy(), equal_nan=True), k
    finally:
        ctx.close()
