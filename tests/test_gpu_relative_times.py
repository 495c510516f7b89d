"""Times of calls with rarely used options, as multiples of the same call's ordinary time on the same GPU: a guard against an
option becoming several times slower than it has to be.  Each limit lies well above the multiple that the option takes
and well below one that it once took, both stated."""
import statistics
import time

import numpy as np
import pytest

import mdz_rheo as R
import mdz_workloads as W
from golden.cases import alloc_point_outputs, point_case

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def on_device(a):
    d = {k: ([torch.from_numpy(x).cuda() for x in v] if isinstance(v, list) else torch.from_numpy(v).cuda())
         for k, v in a.items()}
    torch.cuda.synchronize()
    return d


def kernel_ms(call, reps=9):
    for _ in range(3):
        call()
    return statistics.median(call()[1].elapsed_ms for _ in range(reps))


@pytest.fixture(scope="module")
def ctx():
    c = R.Context(0)
    yield c
    c.close()


def test_power_law_viscoplasticity(ctx):
    """n_vp = 2 against n_vp = 1 at 1025 x 1025 cells: 3.5 times (14 with CUDA's pow in every pass)."""
    w = W.plain_large(seed=3, ncx=1025)
    F = R.FieldSet(on_device(w.arrays))
    plain = kernel_ms(lambda: ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE))
    for p in range(5):
        w.mat.eta_vp[p], w.mat.n_vp[p] = 1e12, 2.0
    power = kernel_ms(lambda: ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE, check=False))
    print("n_vp", power / plain)
    assert power < 6.0 * plain


def test_points_with_the_grain_size_solve(ctx):
    """48,000 points against 12,000 (less than one CTA of 128 per SM): 2.7 times with three CTAs on an SM (3.6 with two)."""
    md, m, pin, aniso, centroid, fu = point_case("gse")

    def seconds(rep):
        n = pin["T"].size * rep
        p, o = on_device({k: np.tile(v, rep) for k, v in pin.items()}), on_device(alloc_point_outputs(n))
        args = R.make_points(p, o, centroid=centroid, final_update=fu)
        t = []
        for _ in range(12):
            t0 = time.perf_counter()
            assert ctx.points(md, m, *args, n, mem=R.MEM_DEVICE) == R.MDZ_OK
            t.append(time.perf_counter() - t0)
        return statistics.median(t[3:])

    few, many = seconds(100), seconds(400)
    print("points", many / few)
    assert many < 3.15 * few


def test_sweep_between_one_and_two_waves(ctx):
    """340 x 340 cells against 310 x 310 (1.2 times the nodes, both two waves of resident CTAs at 7 per SM): 1.1 times
    (1.45 where the larger grid ran 5 CTAs per SM, in three waves)."""
    t = {}
    for n in (310, 340):
        w = W.plain_large(seed=3, ncx=n)
        F = R.FieldSet(on_device(w.arrays))
        t[n] = kernel_ms(lambda: ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE), 25)
    print("340 / 310", t[340] / t[310])
    assert t[340] < 1.3 * t[310]
