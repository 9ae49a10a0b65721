"""itsu_batch_launch inside a caller's graph capture is refused, whether the library has made its own graph
of the batch yet or not, and the context goes on working."""
import numpy as np
import pytest

from itsu import capi, gen, prefilter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs_before", [1, 2, 3, 4])
def test_launch_under_capture_is_refused(runs_before):
    torch = pytest.importorskip("torch")
    events = [gen.pbpb_event(s, n_tracks=300) for s in range(3)]
    stream = torch.cuda.Stream()
    ctx = capi.Context()
    try:
        ctx.set_stream(stream.cuda_stream)
        batch = prefilter.DeviceBatch(ctx, events, torch.device("cuda", 0))
        torch.cuda.synchronize()
        ctx.batch_run(batch.batch)
        want = [ctx.results(e)["roads"].copy() for e in range(len(events))]
        assert sum(map(len, want)) > 0
        for _ in range(runs_before - 1):
            ctx.batch_launch(batch.batch)
            ctx.batch_status()
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream, capture_error_mode="thread_local"):
            with pytest.raises(capi.ItsuError):
                ctx.batch_launch(batch.batch)
        for _ in range(3):
            ctx.batch_launch(batch.batch)
            ctx.batch_status()
            for e, roads in enumerate(want):
                assert np.array_equal(ctx.results(e)["roads"].view(np.uint8), roads.view(np.uint8))
    finally:
        ctx.close()
