"""The statistics a call returns are its own, whatever ran before it on the context: waiting
calls leave the device's counters at their initial values for the next one, calls that do not
wait and captured graphs reset them themselves."""
import pytest

import mdz_rheo as R
import mdz_workloads as W
from common import clone

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def to_device(arrays):
    return {k: ([torch.from_numpy(x).cuda() for x in v] if isinstance(v, list) else torch.from_numpy(v).cuda())
            for k, v in arrays.items()}


def counts(st):
    return (st.phase_calls, st.newton_iters, st.max_newton_iters, st.plastic_calls, st.status, st.error_node,
            st.fp32_steps)


@pytest.mark.parametrize("before", ["sweep", "async", "failing", "batch_graph", "captured"])
def test_statistics_after(before):
    w = W.plain_large(seed=4, ncx=61)
    other = W.plain_large(seed=5, ncx=90)
    bad = W.plain_large(seed=15, ncx=32)
    bad.arrays["d0_n"][77] = 0.0  # diffusion creep at grain size 0
    want_ctx, ctx = R.Context(0), R.Context(0)
    try:
        d, e = to_device(clone(w.arrays)), to_device(clone(other.arrays))
        torch.cuda.synchronize()
        F, G = R.FieldSet(d), R.FieldSet(e)
        want = counts(want_ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE)[1])
        assert want[0] > 0 and want[4] == R.MDZ_OK
        assert counts(ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE)[1]) == want
        if before == "sweep":
            ctx.sweep(other.model, other.mat, G, mem=R.MEM_DEVICE)
        elif before == "async":
            ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE, flags=R.SWEEP_ASYNC)
            for _ in range(2):  # readable as often as it is asked for
                assert counts(ctx.sync()[1]) == want
            ctx.sweep(other.model, other.mat, G, mem=R.MEM_DEVICE, flags=R.SWEEP_ASYNC)
        elif before == "failing":
            rc, st = ctx.sweep(bad.model, bad.mat, R.FieldSet(bad.arrays), check=False)
            assert rc == R.MDZ_EGRAIN_ZERO
            assert counts(ctx.sync()[1]) == counts(st)
        elif before == "batch_graph":
            b = R.Batch(ctx, [other.model], [other.mat], [G])
            b.capture(2)
            assert b.launch()[1].phase_calls > 0
            b.close()
        else:
            s = torch.cuda.Stream()
            ctx.set_stream(s.cuda_stream)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
                ctx.sweep(other.model, other.mat, G, mem=R.MEM_DEVICE, flags=R.SWEEP_ASYNC)
            assert counts(ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE)[1]) == want
            g.replay()
            torch.cuda.synchronize()
        for _ in range(2):
            assert counts(ctx.sweep(w.model, w.mat, F, mem=R.MEM_DEVICE)[1]) == want
            assert counts(ctx.sync()[1]) == want
    finally:
        ctx.close()
        want_ctx.close()
