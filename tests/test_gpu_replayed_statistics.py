"""What mdz_rheo_sync returns after a replay of a caller's graph that holds an MDZ_SWEEP_ASYNC call: the replay's own
status and counts, whatever waiting calls ran on the context since the capture; and a replay starts from reset counters,
the work counter of the persistent sweep among them."""
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


def counts(st):
    return (st.phase_calls, st.newton_iters, st.max_newton_iters, st.plastic_calls, st.fp32_steps, st.status, st.error_node)


def test_replays_start_from_reset_counters():
    good, bad = W.plain_large(seed=4, ncx=61), failing()
    ctx = R.Context(0)
    try:
        F, G = R.FieldSet(on_device(good)), R.FieldSet(on_device(bad))
        want = counts(ctx.sweep(good.model, good.mat, F, mem=R.MEM_DEVICE)[1])
        replay = captured(ctx, lambda: ctx.sweep(good.model, good.mat, F, mem=R.MEM_DEVICE, flags=R.SWEEP_ASYNC))
        for _ in range(3):
            replay()
            assert counts(ctx.sync()[1]) == want
        assert ctx.sweep(bad.model, bad.mat, G, mem=R.MEM_DEVICE, check=False)[0] == R.MDZ_EGRAIN_ZERO
        replay()
        assert counts(ctx.sync()[1]) == want
    finally:
        ctx.close()


def test_replays_of_the_persistent_sweep_update_every_node():
    w = W.plain_large(seed=4, ncx=61)
    d = on_device(w)
    ctx = R.Context(0)
    try:
        ctx.set_launch_shape(False, 128, 8, 2)  # the work-counter form on 8 CTAs
        F = R.FieldSet(d)
        want = counts(ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE)[1])
        eta = d["eta_n"].clone(), d["eta_s"].clone()
        replay = captured(ctx, lambda: ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE, flags=R.SWEEP_ASYNC))
        for _ in range(2):
            d["eta_n"].zero_()
            d["eta_s"].zero_()
            torch.cuda.synchronize()
            replay()
            assert counts(ctx.sync()[1]) == want
            assert torch.equal(d["eta_n"], eta[0]) and torch.equal(d["eta_s"], eta[1])
    finally:
        ctx.close()
