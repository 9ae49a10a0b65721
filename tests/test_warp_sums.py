"""Tile sums of the scans hold 64 bits: counts near 2^31 in every lane, whose sum over a warp passes
2^31 and 2^32, reach the tiles whole (csrc/itsu_kernels.cu add_to_tile, warp_sum), so that the scans'
checks of the total against the 32-bit index range and the capacities see it. A chain count may be
INT_MAX (Tracker.cxx:477-571 counts roads without a bound), as on layers of 91 coincident clusters."""
import numpy as np
import pytest

import warp_emulation

INT_MAX = 2 ** 31 - 1


def _counts():
    rng = np.random.default_rng(7)
    yield "ordinary", rng.integers(0, 100, 32)
    yield "most of INT_MAX", np.full(32, INT_MAX)
    yield "past 2^31", np.full(32, 91 ** 4)
    yield "past 2^32", np.full(32, 215 ** 4 % INT_MAX)
    yield "mixed", np.where(rng.random(32) < 0.5, rng.integers(0, INT_MAX, 32), rng.integers(1, 9, 32))
    yield "one large", np.where(np.arange(32) == 17, INT_MAX, 1)


def _array(name, values):
    return "const long long %s[32] = {%s};" % (name, ",".join("%dll" % v for v in values))


@pytest.mark.parametrize("name, counts", list(_counts()), ids=[n for n, _ in _counts()])
@pytest.mark.parametrize("split", [0, 1, 13, 32])
@pytest.mark.parametrize("active", [0xffffffff, 0x0ff0f00f])
def test_tile_sums_of_a_warp(name, counts, split, active):
    """The lanes' items are consecutive, those of lanes below `split` the last ones of tile 4."""
    first = 5 * 2048 - split
    main = _array("count", counts) + """
      long long partials[8] = {};
      g_active = %#xu;
      warp([&](int lane) { add_to_tile((int64_t *)partials, %d + lane, (int)count[lane]); });
      for (long long p : partials) std::printf("%%lld\\n", p);""" % (active, first)
    got = warp_emulation.run(["kScanThreads", "kScanItems", "kScanTile", "warp_sum", "add_to_tile"], main)
    want = [0] * 8
    for lane in range(32):
        if (active >> lane) & 1:
            want[(first + lane) // 2048] += int(counts[lane])
    assert got == want


@pytest.mark.parametrize("name, counts", list(_counts()), ids=[n for n, _ in _counts()])
def test_warp_sum(name, counts):
    main = _array("count", counts) + """
      unsigned long long sums[32];
      warp([&](int lane) { sums[lane] = warp_sum(0xffffffffu, (unsigned)count[lane]); });
      for (unsigned long long s : sums) std::printf("%llu\\n", s);"""
    assert warp_emulation.run(["warp_sum"], main) == [int(np.sum(counts))] * 32


@pytest.mark.gpu
def test_more_roads_than_indices_is_reported():
    """91 coincident clusters on each layer of one track: 91^4 chains end in each of 91^3 last-layer
    cells, 5e13 roads in all. The run ends in the count overflow error, nothing is written, and the
    context goes on."""
    from itsu import capi, gen
    from oracle import oracle

    ev = gen.make_event(16, 1, pt_mean=3.0, noise=0.0, eta_range=(0.1, 0.2))
    assert [len(l) for l in ev.layers] == [1] * 7
    ctx = capi.Context(device=0)
    try:
        with pytest.raises(capi.ItsuError, match="32-bit index range") as err:
            ctx.clusters_to_tracks([np.repeat(l, 91) for l in ev.layers], ev.vertices[0])
        assert err.value.status == capi.ERR_CAPACITY
        other = gen.pbpb_event(2, 500)
        want = oracle.run_vertex(other.layers, other.vertices[0])
        assert oracle.diff(ctx.run_vertex(other.layers, other.vertices[0]), want) == []
    finally:
        ctx.close()
