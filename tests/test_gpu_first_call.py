"""Calls on a context that holds no buffers yet, or lost some: empty events and batches as the first
call (the passes write offsets and totals of empty runs too), and an ordinary run after one whose
buffers did not fit the device's memory."""
import ctypes

import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu
EMPTY = [np.zeros(0, gen.CLUSTER_DTYPE)] * 7


@pytest.fixture
def ctx():
    c = capi.Context(device=0)
    yield c
    c.close()


def _assert_runs(ctx):
    ev = gen.pp_event(6)
    want = oracle.run_vertex(ev.layers, ev.vertices[0])
    assert oracle.diff(ctx.run_vertex(ev.layers, ev.vertices[0]), want) == []
    assert ctx.clusters_to_tracks(ev.layers, ev.vertices[0]).tobytes() == want["roads"].tobytes()


@pytest.mark.parametrize("staged", [True, False])
def test_vertex_without_clusters(ctx, staged):
    vertex = np.zeros(3, np.float32)
    if staged:
        assert oracle.diff(ctx.run_vertex(EMPTY, vertex), oracle.run_vertex(EMPTY, vertex)) == []
    else:
        assert len(ctx.clusters_to_tracks(EMPTY, vertex)) == 0
    _assert_runs(ctx)


@pytest.mark.parametrize("n_events", [0, 1, 300])
@pytest.mark.parametrize("streamed", [False, True])
def test_batch_without_clusters(n_events, streamed):
    ctx = capi.Context(device=0, flags=capi.FLAG_STREAM_HOST if streamed else 0)
    try:
        offsets, vertices = np.zeros(7 * n_events + 1, np.int32), np.zeros((n_events, 3), np.float32)
        roads, road_offsets = ctx.batch_run_host(np.zeros(0, gen.CLUSTER_DTYPE), offsets, vertices)
        assert len(roads) == 0 and list(road_offsets) == [0] * (n_events + 1)
        _assert_runs(ctx)
    finally:
        ctx.close()


def test_batch_without_events(ctx):
    empty = ctx.batch_device(0, 0, 0, 0, 0)
    ctx.batch_run(empty)
    ctx.batch_launch(empty)
    ctx.batch_status()
    with pytest.raises(capi.ItsuError) as err:
        ctx.batch_run(ctx.batch_device(16, 0, 0, 0, 5))  # clusters of no event: refused before anything runs
    assert err.value.status == capi.ERR_INVALID
    frames = capi.Frames()
    ctx._check(ctx.lib.itsu_frames_run_host(ctx.h, ctypes.byref(frames), None, 0, None))
    _assert_runs(ctx)


def test_run_after_a_failed_growth(ctx):
    """2^31 - 1 clusters need some 700 GB: refused for want of memory before the batch is read."""
    _assert_runs(ctx)
    with pytest.raises(capi.ItsuError) as err:
        ctx.batch_run(ctx.batch_device(16, 16, 16, 1, 2 ** 31 - 1))
    assert err.value.status == capi.ERR_NOMEM
    with pytest.raises(capi.ItsuError) as err:
        ctx.results(0)  # the results went with the buffers
    assert err.value.status == capi.ERR_STATE
    _assert_runs(ctx)
