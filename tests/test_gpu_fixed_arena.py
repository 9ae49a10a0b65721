"""A fixed arena (ITSU_FLAG_NO_GROW) whose five capacities are exactly what the results need runs them,
however many tracklet pairs pass the cell stage's precut. Narrow bundles that miss the vertex have up
to seventy such pairs per tracklet and few cells; their spans take the warp queue, overflow it, or stand
behind outer clusters with more outgoing tracklets than a mask holds."""
import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu


def _bundle(seed, n, spread):
    """n clusters on each of layers 0 to 2, on lines that pass 3 mm beside the vertex; one elsewhere."""
    rng = np.random.default_rng(seed)
    layers, first = [], 0
    for layer, r in enumerate(gen.RADII_CM):
        k = n if layer < 3 else 1
        phi = 2.0 + np.arcsin(0.3 / r) + rng.uniform(-spread, spread, k)
        c = np.zeros(k, gen.CLUSTER_DTYPE)
        c["x"], c["y"], c["z"] = r * np.cos(phi), r * np.sin(phi), 0.3 * r + rng.uniform(-0.02, 0.02, k)
        c["alpha"], c["mc"], c["id"] = phi, rng.integers(0, 99, k), np.arange(first, first + k)
        first += k
        layers.append(c)
    return gen.Event(vertices=np.zeros((1, 3), np.float32), layers=layers, labels=np.zeros(0, gen.LABEL_DTYPE))


@pytest.mark.parametrize("pair_prefilter", [False, True])
@pytest.mark.parametrize("n, n_events, spread", [(20, 64, 0.002), (60, 8, 0.002), (300, 1, 0.002), (300, 2, 0.01)])
def test_exact_capacities_suffice(n, n_events, spread, pair_prefilter):
    events = [_bundle(100 * n + k, n, spread) for k in range(n_events)]
    clusters, offsets, vertices = gen.pack_batch(events)
    model = capi.prefilter_init(5)
    growing = capi.Context()
    fixed = None
    try:
        growing.prefilter_set_model(model)
        growing.prefilter_enable(pair_prefilter)
        roads, road_offsets = growing.batch_run_host(clusters, offsets, vertices)
        want = [growing.results(e) for e in range(n_events)]
        if not pair_prefilter:
            for e in (0, n_events - 1):
                assert oracle.diff(want[e], oracle.run_vertex(events[e].layers, events[e].vertices[0])) == []
        caps = {"max_" + name: max(int(used), 1) for name, used in growing.memory_usage()["used"].items()}
        fixed = capi.Context(flags=capi.FLAG_NO_GROW, max_clusters=len(clusters), max_events=n_events, **caps)
        fixed.prefilter_set_model(model)
        fixed.prefilter_enable(pair_prefilter)
        got, got_offsets = fixed.batch_run_host(clusters, offsets, vertices, roads_capacity=caps["max_roads"])
        assert np.array_equal(got_offsets, road_offsets) and got.tobytes() == roads.tobytes()
        for e in range(n_events):
            assert oracle.diff(fixed.results(e), want[e]) == [], e
        assert oracle.diff(fixed.run_vertex(events[0].layers, events[0].vertices[0]), want[0]) == []
    finally:
        growing.close()
        if fixed is not None:
            fixed.close()


def test_pairs_beyond_a_quarter_of_the_memory():
    """1.36e9 pairs of 4 million tracklets: a growing arena keeps places for some of them and counts the
    cells of the other spans, a fixed one counts nearly all; tracklets, cells and lookups are the same."""
    ev = _bundle(1, 1400, 0.002)
    growing, fixed = capi.Context(), None
    try:
        want = growing.run_vertex(ev.layers, ev.vertices[0])
        assert sum(map(len, want["cells"])) > 1000
        usage = growing.memory_usage()
        assert usage["device_bytes"] < 60e9
        roads = growing.clusters_to_tracks(ev.layers, ev.vertices[0])
        assert oracle.diff(growing.results(0), want) == []
        caps = {"max_" + name: max(int(used), 1) for name, used in usage["used"].items()}
        fixed = capi.Context(flags=capi.FLAG_NO_GROW, max_clusters=sum(map(len, ev.layers)), max_events=1, **caps)
        assert fixed.memory_usage()["device_bytes"] < 2e9
        assert fixed.clusters_to_tracks(ev.layers, ev.vertices[0]).tobytes() == roads.tobytes()
        assert oracle.diff(fixed.results(0), want) == []
    finally:
        growing.close()
        if fixed is not None:
            fixed.close()


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("flags", [0, capi.FLAG_STREAM_HOST])
def test_scratch_overflow_with_event_groups(group, flags):
    """The first group's pairs do not fit the entry scratch of a new arena: the groups after it are
    written and counted all the same, for what the run needs, and the repeated run gives the oracle's
    results."""
    events = [_bundle(7, 180, 0.002)] + [gen.pbpb_event(60 + k) for k in range(3)]
    want = [oracle.run_vertex(ev.layers, ev.vertices[0]) for ev in events]
    clusters, offsets, vertices = gen.pack_batch(events)
    ctx = capi.Context(flags=flags, stream_chunk_clusters=60000)
    try:
        for band in range(32):
            ctx.set_tune(band, 256, 8, 1, group)
        for _ in range(2):
            roads, road_offsets = ctx.batch_run_host(clusters, offsets, vertices)
            for e, w in enumerate(want):
                assert roads[road_offsets[e]:road_offsets[e + 1]].tobytes() == w["roads"].tobytes(), e
        if flags == 0:
            for e, w in enumerate(want):
                assert oracle.diff(ctx.results(e), w) == [], e
    finally:
        ctx.close()
