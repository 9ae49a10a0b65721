"""The clustering's launch shapes: CTAs of 64, 256 and 512 threads and layers split over clusters of 2,
4 and 8 CTAs give the reference's sorted clusters and index tables (PrimaryVertexContext.cxx:31-142)
at the sizes where the shapes change, for empty and one-cluster layers, with negative bins, and for
layers of very different sizes."""
import ctypes

import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu
HALF = (16.333, 16.333, 16.333, 42.140, 42.140, 73.745, 73.745)


def _layers(rng, counts, beyond=0):
    out, first = [], 0
    for layer, n in enumerate(counts):
        c = np.zeros(n, gen.CLUSTER_DTYPE)
        phi = rng.uniform(0.0, 2.0 * np.pi, n)
        c["x"], c["y"] = gen.RADII_CM[layer] * np.cos(phi), gen.RADII_CM[layer] * np.sin(phi)
        c["z"] = rng.uniform(-gen.HALF_LENGTHS_CM[layer], gen.HALF_LENGTHS_CM[layer], n)
        if beyond and n > beyond:  # phi bin 0 beyond -z: negative bins, many of them tied
            at = rng.permutation(n)[:beyond]
            c["x"][at], c["y"][at] = gen.RADII_CM[layer], 0.02 * gen.RADII_CM[layer]
            c["z"][at] = -HALF[layer] - rng.integers(1, 60, beyond)
        c["alpha"] = phi
        c["mc"] = rng.integers(-1, 5000, n)
        c["id"] = np.arange(first, first + n)
        first += n
        out.append(c)
    return out


def _expected(layer, raw, vertex):
    """The layer's clusters transformed by the oracle and stably sorted by bin, and its index table."""
    lib, done = oracle.lib(), np.zeros(len(raw), gen.CLUSTER_DTYPE)
    transform = lib.oracle_transform_cluster
    transform.argtypes, transform.restype = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p], None
    vertex, raw = np.ascontiguousarray(vertex, np.float32), np.ascontiguousarray(raw)
    for k in range(len(raw)):
        transform(layer, vertex.ctypes.data, raw.ctypes.data + 36 * k, done.ctypes.data + 36 * k)
    done = done[np.argsort(done["bin"], kind="stable")]
    table = np.searchsorted(done["bin"], np.arange(401), side="left").astype(np.int32)
    table[0] = 0
    return done, table


CASES = [
    ("tiny", 3, (0, 1, 2, 31, 33, 64, 192), 0),
    ("medium", 2, (193, 512, 5, 1024, 0, 700, 1000), 100),
    ("one event, split eight ways", 1, (1025, 4096, 4097, 9000, 1, 0, 5000), 0),
    ("one event, negative bins", 1, (1500, 2500, 1100, 1200, 1300, 1400, 1600), 700),
    ("split in four", 20, (1030, 1030, 1040, 1025, 1030, 1035, 1026), 0),
    ("split in two", 43, (1100, 1090, 1080, 1100, 1070, 1060, 1100), 300),
    ("uneven, not split", 30, (20, 10, 3000, 15, 0, 30, 5), 0),
]


@pytest.mark.parametrize("name, n_events, counts, beyond", CASES)
def test_sorted_clusters_and_tables(name, n_events, counts, beyond):
    rng = np.random.default_rng(len(name) * 1000 + n_events)
    events = []
    for _ in range(n_events):
        vertex = rng.normal(0.0, [0.005, 0.005, 5.0]).astype(np.float32)[None]
        events.append(gen.Event(vertices=vertex, layers=_layers(rng, counts, beyond), labels=np.zeros(0, gen.LABEL_DTYPE)))
    ctx = capi.Context(device=0)
    try:
        if n_events == 1:
            ctx.initialize(events[0].layers, events[0].vertices[0])
        else:
            clusters, offsets, vertices = gen.pack_batch(events)
            ctx.batch_run_host(clusters, offsets, vertices)
        for e in {0, n_events // 2, n_events - 1}:
            got = ctx.results(e)
            for layer in range(7):
                want, table = _expected(layer, events[e].layers[layer], events[e].vertices[0])
                assert got["clusters"][layer].tobytes() == want.tobytes(), (name, e, layer)
                if layer > 0:
                    assert np.array_equal(got["index_tables"][layer - 1], table), (name, e, layer)
    finally:
        ctx.close()
