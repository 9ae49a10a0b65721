"""The tracklet walk's fixed-point window (csrc/itsu_device.cuh cluster_key, tracklet_window) loses no candidate.

A numpy binary32 restatement of the cluster keys and of the window is compared with the tracklet cut
(Tracker.cxx:93-100) on candidates drawn across a regular layer's clusters and at the edges of each
cut: every cluster that passes the cut must pass the window."""
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = open(os.path.join(ROOT, "tracking-itsu_b200", "csrc", "itsu_device.cuh")).read()
F = np.float32
Z_HALF = np.array([16.333, 16.333, 16.333, 42.140, 42.140, 73.745, 73.745], F)
INV_Z_BIN = (10.0 / Z_HALF.astype(np.float64)).astype(F)
MAX_DZ = np.array([0.1, 0.1, 0.3, 0.3, 0.3, 0.3], F)


def _constant(name):
    m = re.search(r"constexpr float %s = ([0-9.]+)f;" % name, HEADER)
    assert m, name
    return F(m.group(1))


PHI_UNITS, Z_PER_BIN, PHI_CUT = _constant("kKeyPhiUnits"), _constant("kKeyZPerBin"), _constant("kPhiCoordinateCut")
PHI_WRAP = F(float.fromhex(re.search(r"constexpr float kPhiWrapTracklet = (\S+)f;", HEADER).group(1)))


def _to_int(x, rounding):
    """float -> int32 as the device converts: saturating, NaN gives 0."""
    r = rounding(x.astype(np.float64))
    return np.where(np.isnan(r), 0, np.clip(r, -2.0 ** 31, 2.0 ** 31 - 1)).astype(np.int64)


def _key_z(layer, z):
    return _to_int((z + Z_HALF[layer]) * (INV_Z_BIN[layer] * Z_PER_BIN), np.floor)


def _window_pass(layer, phi1, reach, zlo, zhi, z2, phi2):
    spread = _to_int(np.maximum(reach, F(0)) * PHI_UNITS, np.ceil) + 2
    start = np.clip(_key_z(layer, zlo), 1, 65535) - 1
    stop = np.clip(_key_z(layer, zhi), 0, 65534) + 1
    key_phi, key_z = _to_int(phi2 * PHI_UNITS, np.rint) & 0xFFFF, np.clip(_key_z(layer, z2), 0, 65535)
    phi = (key_phi - _to_int(phi1 * PHI_UNITS, np.rint) + spread) & 0xFFFF
    return (phi <= 2 * spread) & (((key_z - start) & 0xFFFF) <= stop - start)


def _nudge(rng, x, ulps=4):
    """x moved by a few representable steps."""
    bits = x.astype(F).view(np.int32).astype(np.int64)
    return (bits + rng.integers(-ulps, ulps + 1, len(x))).astype(np.int32).view(F)


@pytest.mark.parametrize("spread_r", [0.0, 0.016, 2.0])
@pytest.mark.parametrize("layer", range(1, 7))
def test_window_keeps_every_candidate_that_passes_the_cut(layer, spread_r):
    rng = np.random.default_rng(100 * layer + int(10 * spread_r))
    n, radius, two_pi = 200_000, F(3.0 * layer + 1.0), F(6.2831853)
    z_bin = lambda z: _to_int((z + Z_HALF[layer]) * INV_Z_BIN[layer], np.trunc)  # noqa: E731
    passed = 0
    with np.errstate(all="ignore"):
        for edge in ("none", "z", "phi"):
            r1 = rng.uniform(0.5 * radius, radius - 0.5, n).astype(F)
            rmin, rmax = radius, F(radius + F(spread_r))
            r2 = rng.uniform(rmin, rmax, n).astype(F).clip(rmin, rmax)
            z1 = rng.uniform(-Z_HALF[layer], Z_HALF[layer], n).astype(F)
            tan = (3 * rng.uniform(-1, 1, n) ** 3).astype(F)
            phi1 = rng.uniform(0, two_pi, n).astype(F)
            max_dz = MAX_DZ[layer - 1]
            at = tan * (r2 - r1) + z1
            z2 = at + (max_dz * rng.uniform(-1, 1, n)).astype(F)
            phi2 = phi1 + (PHI_CUT * rng.uniform(-1, 1, n)).astype(F)
            side = np.where(rng.integers(0, 2, n) == 0, F(-1), F(1))
            if edge == "z":
                z2 = _nudge(rng, at + side * max_dz)
            if edge == "phi":
                phi2 = _nudge(rng, phi1 + side * PHI_CUT)
            phi2 = np.where(phi2 < 0, phi2 + two_pi, np.where(phi2 >= two_pi, phi2 - two_pi, phi2)).astype(F)
            ok = (z_bin(z2) >= 0) & (z_bin(z2) < 20)  # a regular layer's cluster
            dphi = np.abs(phi1 - phi2)
            cut = ok & (np.abs(tan * (r2 - r1) + z1 - z2) < max_dz) & ((dphi < PHI_CUT) | (dphi > PHI_WRAP))
            p1, p2 = tan * (rmin - r1) + z1, tan * (rmax - r1) + z1
            zlo, zhi = np.minimum(p1, p2) - max_dz - F(1e-3), np.maximum(p1, p2) + max_dz + F(1e-3)
            kept = _window_pass(layer, phi1, np.full(n, PHI_CUT, F), zlo, zhi, z2, phi2)
            assert not (cut & ~kept).any()
            passed += int(cut.sum())
    assert passed > n
