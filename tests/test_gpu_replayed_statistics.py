"""What mdz_rheo_sync returns after a replay of a caller's graph that holds an MDZ_SWEEP_ASYNC call: the replay's own
status and counts, whatever waiting calls ran on the context since the capture."""
import pytest

import mdz_rheo as R
import mdz_workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def on_device(w):
    d = {k: ([torch.from_numpy(x).cuda() for x in v] if isinstance(v, list) else torch.from_numpy(v).cuda())
         for k, v in w.arrays.items()}
    torch.cuda.synchronize()
    return d


def captured(ctx, call):
    s = torch.cuda.Stream()
    ctx.set_stream(s.cuda_stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        call()

    def replay():
        with torch.cuda.stream(s):
            g.replay()
    return replay


def failing():
    w = W.plain_large(seed=15, ncx=32)
    w.arrays["d0_n"][77] = 0.0  # diffusion creep at grain size 0
    return w


@pytest.mark.parametrize("between", ["sweep", "strain_rates"])
def test_sync_reports_the_failure_of_a_replay(between):
    good, bad, vel = W.plain_large(seed=4, ncx=61), failing(), W.velocity_field(seed=9, ncx=40)
    ctx = R.Context(0)
    try:
        F, G, sr = R.FieldSet(on_device(good)), R.FieldSet(on_device(bad)), on_device(vel)
        replay = captured(ctx, lambda: ctx.sweep(bad.model, bad.mat, G, mem=R.MEM_DEVICE, flags=R.SWEEP_ASYNC))
        for _ in range(2):
            if between == "sweep":
                assert ctx.sweep(good.model, good.mat, F, mem=R.MEM_DEVICE)[0] == R.MDZ_OK
            else:
                ctx.strain_rates(vel.model, vel.info["dx"], vel.info["dz"], sr, mem=R.MEM_DEVICE)
            replay()
            rc, st = ctx.sync()
            assert rc == st.status == R.MDZ_EGRAIN_ZERO and st.error_node == 77
    finally:
        ctx.close()


def test_sync_of_a_replay_leaves_no_error_behind():
    """The context's events were recorded by the capture only, so no time can be read from them."""
    vel = W.velocity_field(seed=9, ncx=40)
    sr = on_device(vel)
    ctx = R.Context(0)
    try:
        run = lambda flags: ctx.strain_rates(vel.model, vel.info["dx"], vel.info["dz"], sr, mem=R.MEM_DEVICE, flags=flags)
        replay = captured(ctx, lambda: run(R.SWEEP_ASYNC))
        replay()
        assert ctx.sync()[0] == R.MDZ_OK
        assert run(0)[0] == R.MDZ_OK
    finally:
        ctx.close()
