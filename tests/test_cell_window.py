"""The cell stage's fixed-point precut (csrc/itsu_device.cuh tracklet_key, cell_window) loses no pair.

A numpy binary32 restatement of the keys and of the window is compared with the exact cheap cell
cuts (Tracker.cxx:161-173, csrc/itsu_device.cuh cell_precut_dz) on pairs drawn across the accepted
inputs and on pairs at the edges of each cut: every pair that passes the cuts must pass the window."""
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = open(os.path.join(ROOT, "tracking-itsu_b200", "csrc", "itsu_device.cuh")).read()
F = np.float32
MAX_DZ = np.array([0.2, 0.4, 0.5, 0.6, 3.0], F)


def _constant(name, kind=float):
    m = re.search(r"constexpr (?:float|int) %s = ([0-9a-fA-Fx.p+-]+?)f?;" % name, HEADER)
    assert m, name
    return kind(m.group(1))


TAN_UNITS, PHI_UNITS, REACH = F(_constant("kKeyTanUnits")), F(_constant("kKeyPhiUnits")), _constant("kKeyPhiReach", int)
PHI_WRAP = F(float.fromhex(re.search(r"constexpr float kPhiWrapCell = (\S+)f;", HEADER).group(1)))


def _to_int(x, rounding):
    """float -> int32 as the device converts: saturating, NaN gives 0."""
    r = rounding(x.astype(np.float64))
    return np.where(np.isnan(r), 0, np.clip(r, -2.0 ** 31, 2.0 ** 31 - 1)).astype(np.int64)


def _key(t, phi):
    return ((_to_int(phi * PHI_UNITS, np.rint) & 0xFFFF) << 16) | (_to_int(t * TAN_UNITS, np.rint) & 0xFFFF)


def _window_pass(t1, phi1, z1, r1, vz, max_dz, key2):
    z_beam = t1 * r1
    b = z1 - vz - z_beam
    reach = max_dz + F(1e-5) + F(1e-6) * (np.abs(z_beam) + np.abs(z1) + np.abs(vz) + r1)
    scale = F(2.0) / r1
    near = ~(r1 > F(0.01))
    lo = np.where(near, F(-0.0251), np.fmax(F(-0.0251), (b - reach) * scale))
    hi = np.where(near, F(0.0251), np.fmin(F(0.0251), (b + reach) * scale))
    start, stop = _to_int(lo * TAN_UNITS, np.floor) - 2, _to_int(hi * TAN_UNITS, np.ceil) + 2
    key1 = _key(t1, phi1)
    phi = ((key2 >> 16) - (key1 >> 16) + REACH) & 0xFFFF  # above the lowest, in each half on its own
    tan = ((key2 & 0xFFFF) - (key1 & 0xFFFF) - start) & 0xFFFF
    return (lo <= hi) & (phi <= 2 * REACH) & (tan <= stop - start)


def _cuts(t1, phi1, z1, r1, vz, max_dz, t2, phi2):
    dphi = np.abs(phi1 - phi2)
    dir_z = -(F(0.5) * (t1 + t2)) * r1 + z1
    return (np.abs(t1 - t2) < F(0.025)) & ((dphi < F(0.14)) | (dphi > PHI_WRAP)) & (np.abs(dir_z - vz) < max_dz)


def _nudge(rng, x, ulps=4):
    """x moved by a few representable steps."""
    bits = x.astype(F).view(np.int32).astype(np.int64)
    return (bits + rng.integers(-ulps, ulps + 1, len(x))).astype(np.int32).view(F)


@pytest.mark.parametrize("z_scale, t_scale, r_lo, r_hi", [
    (20.0, 1.2, 2.2, 40.0),       # the tracker's own range
    (20.0, 8.0, 2.2, 40.0),       # steep tracklets
    (1e6, 1e3, 2.2, 40.0),        # the largest accepted coordinates
    (1e6, 2e6, 1e-3, 1e6),        # tanL beyond the keys' saturation
    (1.0, 1e30, 0.0, 0.02),       # clusters on the beam line, overflowing products
])
def test_window_keeps_every_pair_that_passes_the_cuts(z_scale, t_scale, r_lo, r_hi):
    rng = np.random.default_rng(int(t_scale) % 1000 + int(1000 * r_hi) % 997)
    n = 400_000
    passed = 0
    with np.errstate(all="ignore"):
        for edge in ("none", "tan", "z", "phi"):
            max_dz = MAX_DZ[rng.integers(0, 5, n)]
            r1 = rng.uniform(r_lo, r_hi, n).astype(F)
            t1 = (t_scale * rng.uniform(-1, 1, n) ** 3).astype(F)
            vz = rng.uniform(-1, 1, n).astype(F) * F(min(z_scale, 15.0))
            # near the beam line at the vertex, where the delta z cut passes
            z1 = (vz + t1 * r1 + rng.uniform(-1.2, 1.2, n).astype(F) * max_dz).astype(F)
            phi1 = rng.uniform(-np.pi, np.pi, n).astype(F)
            phi1 = np.where(rng.random(n) < 0.2, np.copysign(F(np.pi), phi1), phi1).astype(F)
            t2 = (t1 + rng.uniform(-0.03, 0.03, n).astype(F)).astype(F)
            phi2 = (phi1 + rng.uniform(-0.15, 0.15, n).astype(F)).astype(F)
            if edge == "tan":
                t2 = _nudge(rng, t1 + rng.choice([-0.025, 0.025], n).astype(F))
            elif edge == "z":
                t2 = _nudge(rng, F(2.0) * (z1 - vz + rng.choice([-1.0, 1.0], n).astype(F) * max_dz) / r1 - t1)
            elif edge == "phi":
                phi2 = _nudge(rng, phi1 + rng.choice([-0.14, 0.14], n).astype(F))
            phi2 = np.where(phi2 > np.pi, phi2 - F(2 * np.pi), np.where(phi2 < -np.pi, phi2 + F(2 * np.pi), phi2)).astype(F)
            odd = rng.random(n) < 0.01
            t2 = np.where(odd, rng.choice(np.array([np.nan, np.inf, -np.inf, 0.0], F), n), t2)
            cuts = _cuts(t1, phi1, z1, r1, vz, max_dz, t2, phi2)
            kept = _window_pass(t1, phi1, z1, r1, vz, max_dz, _key(t2, phi2))
            assert not np.any(cuts & ~kept), (edge, int(np.sum(cuts & ~kept)))
            passed += int(np.sum(cuts))
    assert passed > 1000 or t_scale > 1e29
