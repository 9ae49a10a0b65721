"""Grids go by what the host expects of a run (its clusters and the last run's density,
csrc/itsu_capi.cu launch_of), and by nothing else: narrow jets, lines on one another, and ordinary
events in turn through one context, so that every run is launched for the density of another, and
several times each, so that its graph is replayed, give the oracle's results."""
import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu


def _lines(seed, n):
    """n clusters on each of layers 0 to 2 on lines 3 mm beside the vertex (n^2 tracklets between two
    layers), one cluster on the others."""
    rng = np.random.default_rng(seed)
    layers, first = [], 0
    for layer, r in enumerate(gen.RADII_CM):
        k = n if layer < 3 else 1
        phi = 2.0 + np.arcsin(0.3 / r) + rng.uniform(-0.01, 0.01, k)
        c = np.zeros(k, gen.CLUSTER_DTYPE)
        c["x"], c["y"], c["z"] = r * np.cos(phi), r * np.sin(phi), 0.3 * r + rng.uniform(-0.02, 0.02, k)
        c["alpha"], c["mc"], c["id"] = phi, rng.integers(0, 99, k), np.arange(first, first + k)
        first += k
        layers.append(c)
    return gen.Event(vertices=np.zeros((1, 3), np.float32), layers=layers, labels=np.zeros(0, gen.LABEL_DTYPE))


def test_runs_of_changing_density():
    events = [gen.pp_event(1), gen.jet_event(5), gen.make_event(3, 400), _lines(1, 150), gen.pbpb_event(2, 3000), gen.jet_event(6, 40)]
    want = [oracle.run_vertex(ev.layers, ev.vertices[0]) for ev in events]
    ctx = capi.Context(device=0)
    try:
        for order, repeats in (([0, 1, 2, 3, 4, 5], 1), ([5, 3, 0, 4, 1, 2], 4), ([3, 2, 1, 0, 5, 4], 1)):
            for e in order:
                for _ in range(repeats):
                    roads = ctx.clusters_to_tracks(events[e].layers, events[e].vertices[0])
                    assert roads.tobytes() == want[e]["roads"].tobytes(), (order, e)
                assert oracle.diff(ctx.results(0), want[e]) == [], (order, e)
        for e in (1, 0, 3, 2):
            assert oracle.diff(ctx.run_vertex(events[e].layers, events[e].vertices[0]), want[e]) == [], e
        for order in ([1, 1, 5], [0, 2, 4], [3, 1, 4, 0, 2, 5]):
            clusters, offsets, vertices = gen.pack_batch([events[e] for e in order])
            for _ in range(2):
                ctx.batch_run_host(clusters, offsets, vertices)
                for k, e in enumerate(order):
                    assert oracle.diff(ctx.results(k), want[e]) == [], (order, e)
    finally:
        ctx.close()


@pytest.mark.parametrize("chunk", [2000, 30000])
def test_streamed_chunks_of_changing_density(chunk):
    events = [gen.jet_event(5), gen.pp_event(1), gen.make_event(3, 1500), _lines(1, 150), gen.jet_event(6, 60), gen.pbpb_event(2, 3000)] * 2
    want = [oracle.run_vertex(ev.layers, ev.vertices[0])["roads"] for ev in events]
    clusters, offsets, vertices = gen.pack_batch(events)
    ctx = capi.Context(device=0, flags=capi.FLAG_STREAM_HOST, stream_chunk_clusters=chunk)
    try:
        for _ in range(3):
            roads, road_offsets = ctx.batch_run_host(clusters, offsets, vertices)
            for e, exp in enumerate(want):
                assert roads[road_offsets[e]:road_offsets[e + 1]].tobytes() == exp.tobytes(), e
    finally:
        ctx.close()
