"""The pruned tracklet walk reads a row's keys in aligned groups of four into masks of 32 (csrc/itsu_kernels.cu
walk_inner, kMaskKeys). Here one (phi, z) bin per layer holds 28 to 36 or 60 to 68 clusters, with 0 to 3
clusters in front of it, so that every alignment of the first key meets every remainder about one mask
and two; against the oracle."""
import numpy as np
import pytest

from itsu import capi, gen
from oracle import oracle

pytestmark = pytest.mark.gpu
VERTEX = np.array([0.0, 0.0, 0.8], np.float32)


def _event(n, lead):
    """n clusters in one bin of every layer (phi 2.042 is the middle of a row), lead ones in an earlier row."""
    rng = np.random.default_rng(100 * n + lead)
    layers, first = [], 0
    for r in gen.RADII_CM:
        phi = np.concatenate([2.042 + rng.uniform(-0.14, 0.14, n), np.full(lead, 0.05)])
        c = np.zeros(n + lead, gen.CLUSTER_DTYPE)
        c["x"], c["y"] = r * np.cos(phi), r * np.sin(phi)
        c["z"] = np.concatenate([0.8 + rng.uniform(-0.3, 0.3, n), np.full(lead, 0.8)])
        c["alpha"], c["mc"], c["id"] = phi, rng.integers(-1, 99, n + lead), np.arange(first, first + n + lead)
        first += n + lead
        layers.append(c[rng.permutation(n + lead)])
    return layers


@pytest.mark.parametrize("n", list(range(28, 37)) + list(range(60, 69)))
def test_masks_and_remainders(n):
    ctx = capi.Context(device=0)
    try:
        for lead in range(4):
            layers = _event(n, lead)
            want = oracle.run_vertex(layers, VERTEX)
            for c in want["clusters"][1:]:
                assert np.bincount(c["bin"], minlength=400).max() == n
            mismatches = oracle.diff(ctx.run_vertex(layers, VERTEX), want)
            assert mismatches == [], (lead, mismatches[:6])
    finally:
        ctx.close()
