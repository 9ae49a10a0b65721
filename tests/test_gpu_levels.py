"""The level pass's launch shapes (csrc/itsu_kernels.cu level_shape: CTAs of 128 and 512 threads,
clusters of 2, 4 and 8 CTAs, a wide launch per layer) give the reference's neighbour order, levels and
roads (Tracker.cxx:417-571) on both sides of every size where the shape changes."""
import os
import re

import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu
SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tracking-itsu_b200", "csrc", "itsu_kernels.cu")
WIDE = int(re.search(r"constexpr int64_t kWideLevels = (\d+);", open(SOURCE).read()).group(1))


def _event(seed, largest):
    """160 tracks, a third of them in a narrow jet, and on layer 5 clusters far from all to make `largest`."""
    tracks, jet = gen.make_event(seed, 110), gen.jet_event(seed, 50)
    jet.layers[:] = [l.copy() for l in jet.layers]
    rng = np.random.default_rng(seed)
    layers, first = [], 0
    for layer in range(7):
        moved = jet.layers[layer]
        moved["z"] += tracks.vertices[0][2] - jet.vertices[0][2]
        c = np.concatenate([tracks.layers[layer], moved])
        if layer == 5:
            far = np.zeros(largest - len(c), gen.CLUSTER_DTYPE)
            phi = rng.uniform(3.5, 6.0, len(far))
            far["x"], far["y"], far["z"] = gen.RADII_CM[5] * np.cos(phi), gen.RADII_CM[5] * np.sin(phi), rng.uniform(70.0, 73.0, len(far))
            far["mc"] = -1
            c = np.concatenate([c, far])
        c = c[rng.permutation(len(c))]
        c["id"] = np.arange(first, first + len(c))
        first += len(c)
        layers.append(c)
    return gen.Event(vertices=tracks.vertices, layers=layers, labels=tracks.labels)


@pytest.mark.parametrize("n_events, largest", [(1, 192), (1, 193), (2, 682), (2, 683), (2, 1365), (2, 1366), (2, 2730), (2, 2731),
                                               (1, WIDE), (1, WIDE + 1), (3, WIDE + 1), (27, WIDE + 1), (28, WIDE + 1)])
def test_levels_at_the_edges_of_the_shapes(n_events, largest):
    events = [_event(40 + k, largest) for k in range(n_events)]
    assert all(max(map(len, ev.layers)) == largest for ev in events)
    clusters, offsets, vertices = gen.pack_batch(events)
    ctx = capi.Context(device=0)
    try:
        ctx.batch_run_host(clusters, offsets, vertices)
        for e in {0, n_events - 1}:
            want = oracle.run_vertex(events[e].layers, events[e].vertices[0])
            assert len(want["roads"]) > 100
            assert oracle.diff(ctx.results(e), want) == [], e
        want = oracle.run_vertex(events[0].layers, events[0].vertices[0])
        assert oracle.diff(ctx.run_vertex(events[0].layers, events[0].vertices[0]), want) == []
    finally:
        ctx.close()


def test_levels_of_a_large_event():
    """12,500 tracks: the outer layers above the size of the wide launch, 74 thousand cells."""
    ev = gen.make_event(77, 12500)
    assert max(map(len, ev.layers)) > WIDE
    want = oracle.run_vertex(ev.layers, ev.vertices[0])
    ctx = capi.Context(device=0)
    try:
        assert oracle.diff(ctx.run_vertex(ev.layers, ev.vertices[0]), want) == []
        assert ctx.clusters_to_tracks(ev.layers, ev.vertices[0]).tobytes() == want["roads"].tobytes()
    finally:
        ctx.close()
