"""The sweep's register cap at the lines inside its range of sizes (two waves at 5 and at 7 CTAs per SM): no bit changes."""
import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W
from test_gpu_relative_times import on_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aniso", [False, True])
@pytest.mark.parametrize("ncx", [311, 312, 369, 373])
def test_register_cap_keeps_the_bits(aniso, ncx):
    w = W.aniso(seed=3, ncx=ncx) if aniso else W.plain_large(seed=3, ncx=ncx)
    ctx = R.Context(0)
    try:
        fn = ctx.sweep_aniso if aniso else ctx.sweep
        out = []
        for form in (0, 1):
            ctx.set_launch_shape(aniso, 128, 0, form)
            d = on_device(w.arrays)
            fn(w.model, w.mat, R.FieldSet(d), mem=R.MEM_DEVICE)
            out.append(d)
        for k in R.CEN_OUT + R.VER_OUT:
            if out[0].get(k) is not None:
                assert np.array_equal(out[0][k].cpu().numpy(), out[1][k].cpu().numpy(), equal_nan=True), k
    finally:
        ctx.close()
