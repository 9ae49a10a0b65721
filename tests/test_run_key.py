"""A captured graph is only replayed for the event groups it was captured with: the key of a run holds
the groups' cluster ranges (csrc/itsu_capi.cu RunKey, group_bounds), which are launch arguments cut from
the layer offsets on the host. Batches with the same buffers and totals may hold other offsets."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tracking-itsu_b200", "csrc")
SOURCE = open(os.path.join(CSRC, "itsu_capi.cu")).read()

PROGRAM = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <vector>
#define ITSU_LAYERS 7
namespace itsu {
%s
}
%s
%s
static RunKey key(const std::vector<int> &sizes, int group)
{
  std::vector<int32_t> off(1, 0);
  for (int n : sizes) for (int l = 0; l < ITSU_LAYERS; ++l) off.push_back(off.back() + n);
  RunKey k;
  k.n_events = (int32_t)sizes.size();
  k.n_clusters = off.back();
  group_bounds(off.data(), k.n_events, k.n_clusters, group, k.groups);
  return k;
}
int main()
{
  const std::vector<int> a{100, 300, 20, 500, 7}, b{500, 7, 300, 20, 100};
  std::printf("%%d %%d %%d %%d", key(a, 2) == key(a, 2), key(a, 2) == key(b, 2), key(a, 0) == key(b, 0), key(a, 8) == key(b, 8));
}
"""


def test_key_of_another_event_order(tmp_path):
    shapes = "\n".join(re.findall(r"^struct (?:Sort|Level)Shape \{.*?^\};", open(os.path.join(CSRC, "itsu_internal.h")).read(), re.M | re.S))
    struct = re.search(r"^struct RunKey \{.*?^\};", SOURCE, re.M | re.S).group(0)
    bounds = re.search(r"^void group_bounds\(.*?^\}", SOURCE, re.M | re.S).group(0)
    (tmp_path / "key.cpp").write_text(PROGRAM % (shapes, struct, bounds))
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-o", str(tmp_path / "key"), str(tmp_path / "key.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "key")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "0", "1", "1"]  # without groups nothing of the offsets is in the launches


@pytest.mark.gpu
@pytest.mark.parametrize("group", [1, 3, 7])
def test_replays_with_groups(group):
    """Runs of one batch until its graph is replayed, then of its events in other orders."""
    import numpy as np

    from itsu import capi, gen

    events = gen.batch_events(29, n_events=15) + [gen.pp_event(10)]
    plain, grouped = capi.Context(), capi.Context()
    try:
        for b in range(32):
            grouped.set_tune(b, 256, 8, 1, group)
        for order in (list(range(16)), list(range(15, -1, -1)), [5, 0, 9, 1, 15, 3, 2, 14, 4, 6, 13, 7, 12, 8, 11, 10], list(range(16))):
            clusters, offsets, vertices = gen.pack_batch([events[e] for e in order])
            roads, road_offsets = plain.batch_run_host(clusters, offsets, vertices)
            for _ in range(4):
                got, got_offsets = grouped.batch_run_host(clusters, offsets, vertices, roads_capacity=len(roads))
                assert np.array_equal(got_offsets, road_offsets) and got.tobytes() == roads.tobytes()
    finally:
        plain.close()
        grouped.close()
