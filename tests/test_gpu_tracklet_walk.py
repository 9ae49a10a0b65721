"""The pruned tracklet walk (Tracker.cxx:73-113 on regular layers) at the sizes where it can go wrong:
z bins of 0 to a few hundred candidates (group of four, mask of 64 and slot edges, every alignment of
the first key), beside phi = 0 and at the ends of the z range, against the oracle and against the
walk without pruning."""
import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu


def _event(per_patch, phi0, slope, lead):
    """On every layer a patch of per_patch clusters along one direction, and `lead` clusters in front
    of it in the sorted order (phi 0.05, where the patch is elsewhere)."""
    rng = np.random.default_rng(1000 * per_patch + lead)
    layers, first = [], 0
    for layer in range(7):
        r = gen.RADII_CM[layer]
        phi = np.concatenate([phi0 + rng.uniform(-0.35, 0.35, per_patch), np.full(lead, 0.05)])
        z = np.concatenate([slope * r + rng.uniform(-0.25, 0.25, per_patch), np.linspace(-1.0, 1.0, lead) * r])
        n = len(phi)
        c = np.zeros(n, gen.CLUSTER_DTYPE)
        c["x"], c["y"] = r * np.cos(phi), r * np.sin(phi)
        c["z"] = np.clip(z, -0.999 * gen.HALF_LENGTHS_CM[layer], 0.999 * gen.HALF_LENGTHS_CM[layer])
        c["alpha"], c["mc"], c["id"] = phi, rng.integers(-1, 99, n), np.arange(first, first + n)
        first += n
        layers.append(c[rng.permutation(n)])
    return layers


@pytest.mark.parametrize("per_patch", [1, 2, 4, 5, 31, 48, 63, 65, 129, 260])
def test_pruned_walk_matches_oracle(per_patch):
    ctx, vertex = capi.Context(), np.zeros(3, np.float32)
    try:
        for k, (phi0, slope) in enumerate([(2.0, 0.3), (0.1, -0.8), (6.2, 1.8), (3.3, -1.7)]):
            layers = _event(per_patch, phi0, slope, k)
            want = oracle.run_vertex(layers, vertex)
            band = ctx.lib.itsu_multiplicity_band(sum(map(len, layers)), 1)
            for prune in (1, 0):
                ctx.set_tune(band, 256, 8, prune)
                mismatches = oracle.diff(ctx.run_vertex(layers, vertex), want)
                assert mismatches == [], (phi0, prune, mismatches[:6])
    finally:
        ctx.close()
