"""Runs warp-level device functions of the kernels' sources on the CPU.

The named functions are taken from a source file as they stand, compiled as host C++ with the warp
intrinsics below, and run for the 32 lanes of one warp: a lane stops at the first collective whose
result is not known yet, the collective is resolved from all lanes' arguments, and the lanes run
again from the start. Atomic additions take effect once, in the run in which every lane ends."""
import os
import re
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tracking-itsu_b200", "csrc")

PRELUDE = r"""
#include <array>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <utility>
#include <vector>
#define __device__
#define __forceinline__ inline
struct uint2 { unsigned x, y; };
static struct { int x; } threadIdx;
static unsigned g_active = 0xffffffffu;

struct Pending {};
enum Kind { kMatch, kAdd, kShfl, kUp };
struct Call { bool here; Kind kind; unsigned mask; uint32_t value; int arg; };
static std::array<Call, 32> g_calls;
static std::vector<std::array<uint32_t, 32>> g_results;
static size_t g_at;
static std::vector<std::pair<unsigned long long *, unsigned long long>> g_adds;

static uint32_t collective(Kind kind, unsigned mask, uint32_t value, int arg)
{
  const int lane = threadIdx.x & 31;
  if (g_at < g_results.size()) return g_results[g_at++][lane];
  g_calls[lane] = Call{true, kind, mask, value, arg};
  throw Pending();
}

static void resolve()
{
  std::array<uint32_t, 32> r{};
  for (int l = 0; l < 32; ++l) {
    const Call &c = g_calls[l];
    if (!c.here) continue;
    for (int o = 0; o < 32; ++o) {
      if (!((c.mask >> o) & 1u)) continue;
      if (!g_calls[o].here || g_calls[o].kind != c.kind) { std::puts("divergent collective"); std::exit(1); }
      if (c.kind == kMatch && g_calls[o].value == c.value) r[l] |= 1u << o;
      if (c.kind == kAdd) r[l] += g_calls[o].value;
    }
    if (c.kind == kShfl) r[l] = g_calls[c.arg & 31].value;
    if (c.kind == kUp) r[l] = l >= c.arg ? g_calls[l - c.arg].value : c.value;
  }
  g_results.push_back(r);
}

static unsigned __activemask() { return g_active; }
static unsigned __match_any_sync(unsigned mask, unsigned v) { return collective(kMatch, mask, v, 0); }
static unsigned __reduce_add_sync(unsigned mask, unsigned v) { return collective(kAdd, mask, v, 0); }
template <class T> T __shfl_sync(unsigned mask, T v, int from) { return (T)collective(kShfl, mask, (uint32_t)v, from); }
template <class T> T __shfl_up_sync(unsigned mask, T v, int by) { return (T)collective(kUp, mask, (uint32_t)v, by); }
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
static void atomicAdd(unsigned long long *p, unsigned long long v) { g_adds.emplace_back(p, v); }

// f(lane) for every lane of g_active.
template <class F> void warp(F f)
{
  g_results.clear();
  for (;;) {
    bool pending = false;
    g_adds.clear();
    for (int lane = 0; lane < 32; ++lane) {
      g_calls[lane].here = false;
      if (!((g_active >> lane) & 1u)) continue;
      threadIdx.x = lane;
      g_at = 0;
      try { f(lane); } catch (const Pending &) { pending = true; }
    }
    if (!pending) break;
    resolve();
  }
  for (auto &a : g_adds) *a.first += a.second;
}
"""


def function_text(name, text):
    """The definition of the function (or the constant) as the source has it."""
    m = re.search(r"^(?:constexpr [^;\n]*\b%s\b[^;]*;|(?:template <[^>]*>\n)?__device__ [^;{]*\b%s\([^;{]*\)\s*\{.*?^\})" % (name, name), text, re.M | re.S)
    assert m, "no definition of %s" % name
    return m.group(0)


def run(names, main, source="itsu_kernels.cu"):
    """The numbers that `main` prints, with the named definitions of the source in front of it."""
    text = open(os.path.join(CSRC, source)).read()
    program = "\n".join([PRELUDE] + [function_text(n, text) for n in names] + ["int main()\n{\n%s\n}\n" % main])
    with tempfile.TemporaryDirectory() as tmp:
        src, exe = os.path.join(tmp, "warp.cpp"), os.path.join(tmp, "warp")
        with open(src, "w") as f:
            f.write(program)
        subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-w", "-o", exe, src], check=True)
        out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [int(x) for x in out.split()]
