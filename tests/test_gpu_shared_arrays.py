"""Sweeps whose caller passes one device array as an input and an output: the centroids are all updated before the first
vertex, so the vertices see what the centroids wrote, bit for bit in every run."""
import pytest

import mdz_rheo as R
import mdz_workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

PAIRS = {"p_corr": "p_in", "d_n": "d0_n"}


def workload(aniso, ncx):
    w = W.aniso(seed=5, ncx=ncx) if aniso else W.plain_large(seed=5, ncx=ncx)
    for s in "ns":  # a dilatant return, so that p_corr differs from p_in
        w.arrays["dil_" + s][:] = 10.0 * W.DEG
        w.arrays["bet_" + s][:] = 1e-11
    return w


def on_device(w):
    return {k: ([torch.from_numpy(x).cuda() for x in v] if isinstance(v, list) else torch.from_numpy(v).cuda())
            for k, v in w.arrays.items()}


@pytest.mark.parametrize("aniso", [False, True])
@pytest.mark.parametrize("ncx", [40, 300, 520])
def test_vertices_follow_the_centroids(aniso, ncx):
    w = workload(aniso, ncx)
    a, b = on_device(w), on_device(w)
    for out, inp in PAIRS.items():
        b[out] = b[inp]
    torch.cuda.synchronize()
    ctx = R.Context(0)
    try:
        sweep = ctx.sweep_aniso if aniso else ctx.sweep
        sweep(w.model, w.mat, R.FieldSet(a), mem=R.MEM_DEVICE)
        centroids = {k: a[k].clone() for k in R.CEN_OUT if a.get(k) is not None}
        assert not torch.equal(a["p_corr"], a["p_in"])
        for out, inp in PAIRS.items():  # the vertices of a second sweep, from the first one's outputs
            a[inp].copy_(a[out])
        torch.cuda.synchronize()
        sweep(w.model, w.mat, R.FieldSet(a), mem=R.MEM_DEVICE)
        sweep(w.model, w.mat, R.FieldSet(b), mem=R.MEM_DEVICE)
        for k, v in centroids.items():
            assert torch.equal(b[k], v), k
        for k in R.VER_INTERP + R.VER_OUT:
            if a.get(k) is not None:
                assert torch.equal(b[k], a[k]), k
    finally:
        ctx.close()
