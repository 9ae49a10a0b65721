"""The cell count pass's spans of 32, 64 and 128 first tracklets (csrc/itsu_kernels.cu span_of) with all
ways through a span among them: pairs in the warp queue, more pairs than it holds without a crowded outer
cluster, and crowded outer clusters (a jet). Every output of these events equals the oracle's."""
import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu


def _bundle(seed, n):
    """n clusters per layer whose pairs nearly all pass the precut: 32 first tracklets have about 16 n of
    them, more than the queue's 512, while no cluster has more than the 64 outgoing tracklets of a mask."""
    rng = np.random.default_rng(seed)
    layers, first = [], 0
    for layer, r in enumerate(gen.RADII_CM):
        k = n if layer < 4 else 1
        phi = 2.0 + np.arcsin(0.3 / r) + rng.uniform(-0.01, 0.01, k)
        c = np.zeros(k, gen.CLUSTER_DTYPE)
        c["x"], c["y"], c["z"] = r * np.cos(phi), r * np.sin(phi), 0.3 * r + rng.uniform(-0.02, 0.02, k)
        c["alpha"], c["mc"], c["id"] = phi, rng.integers(0, 99, k), np.arange(first, first + k)
        first += k
        layers.append(c)
    return gen.Event(vertices=np.zeros((1, 3), np.float32), layers=layers, labels=np.zeros(0, gen.LABEL_DTYPE))


@pytest.mark.parametrize("background, least, below", [(0, 0, 1 << 20), (4, 1 << 20, 1 << 22), (14, 1 << 22, 1 << 31)])
def test_spans_with_queued_unqueued_and_crowded_pairs(background, least, below):
    jet, bundle, sparse = gen.jet_event(5), _bundle(3, 60), gen.make_event(8, 700)
    central = [gen.pbpb_event(50 + k) for k in range(background)]
    events = central[: background // 2] + [sparse, jet, bundle] + central[background // 2:]
    clusters, offsets, vertices = gen.pack_batch(events)
    ctx = capi.Context(device=0)
    try:
        ctx.batch_run_host(clusters, offsets, vertices)
        assert least <= ctx.memory_usage()["used"]["tracklets"] < below
        for e, ev in enumerate(events):
            if any(ev is own for own in (jet, bundle, sparse)) or e in (0, len(events) - 1):
                want = oracle.run_vertex(ev.layers, ev.vertices[0])
                assert oracle.diff(ctx.results(e), want) == [], e
                if ev is bundle:
                    assert max(np.bincount(t["c1"]).max() for t in want["tracklets"] if len(t)) <= 64
    finally:
        ctx.close()
