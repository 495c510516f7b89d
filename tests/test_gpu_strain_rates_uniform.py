"""Strain rates of flows with exact zeros (rest, rigid blocks, pure and simple shear) on the GPU against the oracle, bit for
bit, the signs of zeros among them; and what they cost beside a flow without zeros."""
import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W
import oracle_lib as O
from test_gpu_relative_times import kernel_ms, on_device

pytestmark = pytest.mark.gpu


def flow(kind, n, air=0.0):
    w = W.velocity_field(seed=9, ncx=n, air=air)
    nx = n + 1
    u, v = w.arrays["u_in"].reshape(n + 2, nx), w.arrays["v_in"].reshape(nx, n + 2)
    if kind == "rest":
        u[:], v[:] = 0.0, 0.0
    elif kind == "negative_zero":
        u[:], v[:] = -0.0, 0.0
    elif kind == "uniform":
        u[:], v[:] = 1e-9, -2e-9
    elif kind == "block":
        u[:, nx // 2:], v[:, nx // 2:] = 1e-9, 0.0
    elif kind == "pure_shear":
        u[:] = 1e-14 * w.info["dx"] * np.arange(nx)[None, :]
        v[:] = -1e-14 * w.info["dz"] * np.arange(nx)[:, None]
    elif kind == "simple_shear":
        u[:], v[:] = 1e-14 * w.info["dz"] * np.arange(n + 2)[:, None], 0.0
    return w


@pytest.fixture(scope="module")
def ctx():
    c = R.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kind", ["rest", "negative_zero", "uniform", "block", "pure_shear", "simple_shear"])
@pytest.mark.parametrize("oop,comp,air", [(0, 0.0, 0.0), (1, 1.0, 0.3)])
def test_same_bits_as_the_oracle(ctx, kind, oop, comp, air):
    w = flow(kind, 70, air)
    ref = {k: v.copy() for k, v in w.arrays.items()}
    assert O.orc_strain_rates(w.model, w.info["dx"], w.info["dz"], ref, oop, comp) == R.MDZ_OK
    d = on_device(w.arrays)
    ctx.strain_rates(w.model, w.info["dx"], w.info["dz"], d, out_of_plane=oop, compressible=comp, mem=R.MEM_DEVICE)
    for k in R.SR_N + R.SR_S:
        assert np.array_equal(d[k].cpu().numpy().view(np.uint64), ref[k].view(np.uint64)), k


def test_time_at_rest(ctx):
    """1025 x 1025 cells at rest against a flow without zeros: 1.7 times (4.2 with the general division and scaling)."""
    t = {}
    for kind in ("noise", "rest"):
        w = flow(kind, 1025)
        d = on_device(w.arrays)
        t[kind] = kernel_ms(lambda: ctx.strain_rates(w.model, w.info["dx"], w.info["dz"], d, mem=R.MEM_DEVICE))
    print("rest", t["rest"] / t["noise"])
    assert t["rest"] < 2.8 * t["noise"]
