"""Cell entries are addressed beyond 2^31: the prefilter and write passes find every entry of spans
whose entries lie anywhere in a scratch of up to 2^32 of them (csrc/itsu_kernels.cu span_entry). The
count pass reserves a place per pair that its precut lets through, so their number is not bounded by
the cells' 32-bit range."""
import numpy as np
import pytest

import warp_emulation

MOST = 2 ** 32 - 64  # entries the scratch may hold


def _spans():
    rng = np.random.default_rng(3)
    ordinary = rng.integers(0, 40, 32)
    yield "from zero", np.cumsum(ordinary) - ordinary, ordinary
    yield "across 2^31", 2 ** 31 - 300 + np.cumsum(ordinary) - ordinary, ordinary
    yield "at the end", MOST - int(ordinary.sum()) + np.cumsum(ordinary) - ordinary, ordinary
    yield "scattered", rng.permutation(32) * 2 ** 27, rng.integers(0, 3, 32) * rng.integers(0, 2 ** 20, 32)
    crowded = np.where(np.arange(32) == 5, 2 ** 31 + 7, np.where(np.arange(32) == 9, 2 ** 30, 1))
    yield "one span of 2^31", np.cumsum(crowded) - crowded, crowded


@pytest.mark.parametrize("name, first, count", list(_spans()), ids=[n for n, _, _ in _spans()])
def test_entries_of_a_warp(name, first, count):
    ends = np.cumsum(count)
    total = int(ends[-1])
    at = sorted({0, total - 1, total // 2, total // 3} | {int(e) + d for e in ends for d in (-1, 0, 1) if 0 <= e + d < total})
    at = [p & ~31 for p in at]  # the passes take 32 consecutive entries at a time
    main = """
      const unsigned first[32] = {%s}, count[32] = {%s};
      static const unsigned tile[] = {%s};
      for (unsigned p0 : tile) {
        long long place[32];
        unsigned sum[32];
        warp([&](int lane) {
          unsigned total;
          const unsigned excl = warp_exclusive_sum(count[lane], total);
          int owner;
          sum[lane] = total;
          place[lane] = span_entry(first[lane], excl, p0 + lane, owner);
        });
        for (int lane = 0; lane < 32; ++lane) if (p0 + lane < sum[lane]) std::printf("%%lld ", place[lane]);
      }""" % (",".join("%du" % v for v in first), ",".join("%du" % v for v in count), ",".join("%du" % p for p in at))
    got = warp_emulation.run(["warp_exclusive_sum", "owner_of", "span_entry"], main)
    want = []
    for p0 in at:
        for p in range(p0, min(p0 + 32, total)):
            owner = int(np.searchsorted(ends, p, side="right"))
            want.append(int(first[owner]) + p - int(ends[owner] - count[owner]))
    assert got == want
