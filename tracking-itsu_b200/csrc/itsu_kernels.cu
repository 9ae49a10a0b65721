// itsu_kernels.cu - sm_100a kernels of the ITS CA track finder.
//
// Every stage is a deterministic count -> exclusive scan -> write sequence over flat,
// event-major arrays, so the output order is the reference's emission order (where a count pass
// uses atomics, to reserve scratch or fill neighbour rows, the write pass restores the order):
//   clustering   a CTA or a cluster of CTAs per (event, layer): vertex-relative transform, stable
//                counting sort by bin (per-warp histograms, warp-match ranks), index table, a
//                4-byte key per cluster for the tracklet pruning (PVC.cxx:31-142)
//   tracklets    count: one thread per inner cluster walking the reference's bin window through a
//                fixed-point window on the keys (Tracker.cxx:45-117); write: a map over tracklets
//                (slope and correctly rounded azimuth), with the lookup table
//   cells        count: the tracklet pairs inside a fixed-point window queued, then the exact cuts
//                and the geometry, a lane per queued pair, one 40-byte entry per found cell
//                (Tracker.cxx:120-235); learned form: the prefilter scores the entries; write: the
//                entries copied to their scanned places, with the lookup table
//   neighbours   one thread per cell walking the next-layer cells of its outer tracklet; rows
//                keyed by the next-layer cell, sorted ascending (Tracker.cxx:417-474)
//   levels       layer-ordered longest-chain DP plus the number of level-decreasing chains; one launch
//                of a CTA cluster per event, or wide ones per layer for few large events
//   roads        one lane per road: the root's k-th chain in the reference's order, Moore-vote
//                labels (Tracker.cxx:477-652)
// Capacity overflow never writes out of bounds: the passes check the scanned totals and scratch
// reservations against the arena capacities, record the requirement and skip; the host grows
// and re-runs.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>

#include "itsu_device.cuh"
#include "itsu_internal.h"
#include "itsu_mlp.cuh"

namespace itsu {
namespace {

constexpr int kThreads = 256;     // threads per block of the fixed-shape helper kernels
constexpr int kMaxThreads = 512;  // upper bound of the tunable per-item kernels' block size
constexpr int kBuckets = kTableSize + 1;  // bucket 0: negative bins; bucket b+1: bin b
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
// The tracklet and cell count passes add each warp's total to the tile sum of the warp's first
// item, which is only right if no warp straddles two tiles: whole warps (block sizes are
// multiples of 32, checked at launch) over tiles of a whole number of warps.
static_assert(kScanTile % 32 == 0, "a warp's 32 items lie in one scan tile");
constexpr float kMaxAbsCoordinate = 1.0e6f;

__device__ __forceinline__ bool capacity_failed(const DevStatus *s) { return (*(volatile const int32_t *)&s->flags & kCapacityMask) != 0; }

__device__ __forceinline__ int grid_threads() { return gridDim.x * blockDim.x; }
__device__ __forceinline__ int64_t global_thread() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }

// A 128-byte line on its way into L2.
__device__ __forceinline__ void prefetch_line(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ------------------------------------------------------------------------------------------
// status

// Status reset of a run; the tracklet scan's tile sums start at zero too (the tracklet count
// pass adds each warp's tracklets to them).
__global__ void k_status_init(Arena a)
{
  if (a.scan_partials) {
    for (int64_t t = global_thread(); t < (a.n_clusters + kScanTile - 1) / kScanTile; t += grid_threads()) {
      a.scan_partials[t] = 0;
    }
  }
  if (global_thread() != 0) {
    return;
  }
  DevStatus *s = a.status;
  s->flags = 0;
  s->invalid_index = INT_MAX;
  s->invalid_event = INT_MAX;
  for (int k = 0; k < 4; ++k) {
    s->total[k] = 0;
  }
  s->cell_entries = 0;
  s->cell_spans = 0;
  s->cell_next = 0;
  s->cell_exact = 0;
  s->trk_crowded = 0;
}

// A launch shape the per-item passes cannot run: the run stops and reports it.
__global__ void k_flag_bad_launch(DevStatus *s) { atomicOr(&s->flags, kFlagLaunchShape); }

// ------------------------------------------------------------------------------------------
// exclusive scan of int32 counts (the count passes fill the scans' tile sums)

__device__ __forceinline__ int64_t scan_length(const int64_t *n_dev, int64_t n_host) { return n_dev ? *n_dev : n_host; }

template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T *warp_totals, T &block_total)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) {
      inc += t;
    }
  }
  if (lane == 31) {
    warp_totals[warp] = inc;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    T w = lane < nw ? warp_totals[lane] : T(0);
    T winc = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const T t = __shfl_up_sync(0xffffffffu, winc, d);
      if (lane >= d) {
        winc += t;
      }
    }
    if (lane < nw) {
      warp_totals[lane] = winc - w;
    }
    if (lane == nw - 1) {
      warp_totals[32] = winc;
    }
  }
  __syncthreads();
  const T res = warp_totals[warp] + inc - v;
  block_total = warp_totals[32];
  __syncthreads();
  return res;
}

// The sum of v over the lanes of mask, in 64 bits: counts go up to INT_MAX each (chains of cells, outer
// clusters in one window), so a warp's sum can pass 2^32. Two 32-bit reductions, of the low and the high
// halves, whose sums stay below 2^21.
__device__ __forceinline__ unsigned long long warp_sum(unsigned mask, unsigned v)
{
  const unsigned long long low = __reduce_add_sync(mask, v & 0xffffu), high = __reduce_add_sync(mask, v >> 16);
  return low + (high << 16);
}

// Adds count (not negative) to the tile sum of item `at`: one atomic for the lanes that are here together
// and whose items lie in one tile.
__device__ __forceinline__ void add_to_tile(int64_t *partials, int64_t at, int count)
{
  const unsigned tile = (unsigned)(at / kScanTile);
  const unsigned peers = __match_any_sync(__activemask(), tile);
  const unsigned long long sum = warp_sum(peers, (unsigned)count);
  if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&partials[tile]), sum);
  }
}

// One kernel per scan: the count passes have added each tile's counts up (partials), and a block
// sums the tile sums before its tiles itself (at most a few thousand of them, from L2) instead of
// taking them from a kernel of its own. The last tile's block checks the total. own_flag: the
// capacity flag this scan may raise, which must not stop its own later blocks (the offsets are kept
// when the stage's outputs are grown). kCellSegments: the grid's last block turns the segments' cell
// counts into cell_seg meanwhile.
__device__ void cell_segments(const Arena &a, int64_t *warp_totals);

template <bool kCellSegments>
__global__ void __launch_bounds__(kScanThreads) k_scan(Arena a, const int32_t *__restrict__ in, int32_t *__restrict__ out,
                                                       const int64_t *n_dev, int64_t n_host, const int64_t *__restrict__ partials,
                                                       int64_t *total_out, int64_t cap, int32_t own_flag)
{
  __shared__ int64_t warp_totals[33];
  DevStatus *const status = a.status;
  if ((*(volatile const int32_t *)&status->flags & kCapacityMask & ~own_flag) != 0) {
    return;
  }
  int blocks = gridDim.x;
  if constexpr (kCellSegments) {
    --blocks;
    if ((int)blockIdx.x == blocks) {
      cell_segments(a, warp_totals);
      return;
    }
  }
  const int64_t n = scan_length(n_dev, n_host);
  const int64_t tiles = max((n + kScanTile - 1) / kScanTile, (int64_t)1);  // an empty scan has a total too
  int64_t before = 0, summed = 0;  // the sum of the tiles below `summed`
  for (int64_t t = blockIdx.x; t < tiles; t += blocks) {
    int64_t part = 0, total;
    for (int64_t k = summed + threadIdx.x; k < t; k += kScanThreads) {
      part += partials[k];
    }
    block_exclusive_scan<int64_t>(part, warp_totals, total);
    before += total;
    summed = t;
    const int64_t base = t * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    if (base + kScanItems <= n) {
      const int4 p = *reinterpret_cast<const int4 *>(in + base);
      const int4 q = *reinterpret_cast<const int4 *>(in + base + 4);
      v[0] = p.x, v[1] = p.y, v[2] = p.z, v[3] = p.w, v[4] = q.x, v[5] = q.y, v[6] = q.z, v[7] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
      }
    }
    int64_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      sum += v[k];
    }
    int64_t run = before + block_exclusive_scan<int64_t>(sum, warp_totals, total);
    int32_t o[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      o[k] = (int32_t)run;
      run += v[k];
    }
    if (base + kScanItems <= n) {
      *reinterpret_cast<int4 *>(out + base) = make_int4(o[0], o[1], o[2], o[3]);
      *reinterpret_cast<int4 *>(out + base + 4) = make_int4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) {
          out[base + k] = o[k];
        }
      }
    }
    if (t == tiles - 1 && threadIdx.x == 0) {
      const int64_t all = before + total;
      *total_out = all;
      out[n] = (int32_t)all;
      if (all > INT_MAX) {
        atomicOr(&status->flags, kFlagCountOverflow);
      }
      if (all > cap) {
        atomicOr(&status->flags, own_flag);
      }
    }
  }
}

// Blocks of a grid-stride kernel: those of a full grid, or what about `items` items need (Launch::tracklets
// and ::cells; any grid gives the same results). A pp event's kernels took 5.5 us each with full grids of
// idle blocks, 4.3 with its own.
unsigned blocks_for(int64_t full, int64_t items, int64_t per_block)
{
  return (unsigned)std::max<int64_t>(1, std::min(full, (items + per_block - 1) / per_block));
}

// The four scans of a run: tracklets per cluster, cells per span of tracklets, neighbours per cell,
// roads per cell. The first leaves the check of its capacity to the segment pass.
template <int kWhich>
void step_scan(const Arena &a, const Launch &l)
{
  switch (kWhich) {
  case 0:
    k_scan<false><<<blocks_for(l.num_sms * 4, a.n_clusters, kScanTile), kScanThreads, 0, l.stream>>>(a, a.trk_count, a.trk_off, nullptr, a.n_clusters, a.scan_partials,
                                                                &a.status->total[kTracklets], INT64_MAX, 0);
    break;
  case 1:
    k_scan<true><<<blocks_for(l.num_sms * 4, l.tracklets / 32, kScanTile) + 1, kScanThreads, 0, l.stream>>>(a, a.cell_span_count, a.cell_span_off, &a.status->cell_spans, 0, a.scan_partials,
                                                               &a.status->total[kCells], a.cap_cells, kFlagCapCells);
    break;
  case 2:
    k_scan<false><<<blocks_for(l.num_sms * 4, l.cells, kScanTile), kScanThreads, 0, l.stream>>>(a, a.nb_count, a.nb_off, &a.status->total[kCells], 0, a.scan_partials,
                                                                &a.status->total[kNeighbours], a.cap_neighbours, kFlagCapNeighbours);
    break;
  default:
    k_scan<false><<<blocks_for(l.num_sms * 4, l.cells, kScanTile), kScanThreads, 0, l.stream>>>(a, a.road_count, a.road_off, &a.status->total[kCells], 0, a.road_partials,
                                                                &a.status->total[kRoads], a.cap_roads, kFlagCapRoads);
  }
}

// ------------------------------------------------------------------------------------------
// (a) clustering: PrimaryVertexContext::initialize (PrimaryVertexContext.cxx:31-142)

__device__ __forceinline__ int bucket_of(int bin) { return bin < 0 ? 0 : bin + 1; }

// A warp's 32 consecutive 36-byte clusters move between global and shared memory as 288 words,
// each load or store instruction covering 128 contiguous bytes; a lane then reads or writes its
// own record in the stage (word stride 9, odd: no bank conflicts).
constexpr int kClusterWords = sizeof(itsu_cluster) / 4;
static_assert(sizeof(itsu_cluster) == 36 && alignof(itsu_cluster) == 4, "cluster layout");

__device__ __forceinline__ void stage_in(int32_t *stage, const itsu_cluster *src, int count)
{
  const int32_t *w = reinterpret_cast<const int32_t *>(src);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kClusterWords; ++k) {
    const int at = k * 32 + lane;
    if (at < count * kClusterWords) {
      stage[at] = w[at];
    }
  }
  __syncwarp();
}

__device__ __forceinline__ void stage_out(itsu_cluster *dst, const int32_t *stage, int count)
{
  __syncwarp();
  int32_t *w = reinterpret_cast<int32_t *>(dst);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kClusterWords; ++k) {
    const int at = k * 32 + lane;
    if (at < count * kClusterWords) {
      w[at] = stage[at];
    }
  }
}

// The 24-byte input record (itsu_cluster_in) in 4-byte words.
constexpr int kClusterInWords = sizeof(itsu_cluster_in) / 4;
static_assert(sizeof(itsu_cluster_in) == 24 && alignof(itsu_cluster_in) == 4, "input record layout");
static_assert(sizeof(itsu_cluster_track) == 16, "track record layout");

// A warp's 32 consecutive records of kWords words each, moved into its stage with coalesced loads.
template <int kWords, typename Record>
__device__ __forceinline__ void stage_in_words(int32_t *stage, const Record *src, int count)
{
  const int32_t *w = reinterpret_cast<const int32_t *>(src);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kWords; ++k) {
    const int at = k * 32 + lane;
    if (at < count * kWords) {
      stage[at] = w[at];
    }
  }
  __syncwarp();
}

// A lane's 24-byte input record from the stage, as a cluster whose phi, r and bin clustering fills.
__device__ __forceinline__ itsu_cluster stage_get_in(const int32_t *stage, int lane)
{
  const int32_t *w = stage + lane * kClusterInWords;  // word stride 6: each access a 2-way bank conflict at most
  itsu_cluster c;
  c.x = __int_as_float(w[0]);
  c.y = __int_as_float(w[1]);
  c.z = __int_as_float(w[2]);
  c.phi = 0.0f;
  c.r = 0.0f;
  c.cluster_id = w[3];
  c.alpha = __int_as_float(w[4]);
  c.mc_id = w[5];
  c.bin = 0;
  return c;
}

__device__ __forceinline__ itsu_cluster stage_get(const int32_t *stage, int lane)
{
  itsu_cluster c;
  int32_t *w = reinterpret_cast<int32_t *>(&c);
#pragma unroll
  for (int k = 0; k < kClusterWords; ++k) {
    w[k] = stage[lane * kClusterWords + k];
  }
  return c;
}

__device__ __forceinline__ void stage_put(int32_t *stage, int lane, const itsu_cluster &c)
{
  const int32_t *w = reinterpret_cast<const int32_t *>(&c);
#pragma unroll
  for (int k = 0; k < kClusterWords; ++k) {
    stage[lane * kClusterWords + k] = w[k];
  }
}

// One segment (event, layer) per cluster of CTAs (of one, where a run has segments enough for the
// chip). Every hit is touched twice: pass 1 reads it in input order and leaves the transformed record
// (32 bytes) in a.sort_recs, pass 4 gathers the records in sorted order and writes every output,
// coalesced. Between them, ranking by bucket and by bin works on indices alone, kept in a.sort_index
// (8 bytes per hit, written and read within the CTA's turn, so mostly L2 hits; kept in shared memory
// instead they cost a CTA per SM on large segments: 0.37 against 0.30 ms per 64 events of 7000
// tracks). Bound by the latency of its barrier-separated phases: 0.30 ms per 128 central events; 0.39
// when it also listed each bin's clusters by z for the tracklet walk, and then 0.41 at two CTAs of 512
// threads per SM in place of three, 0.51 with CTAs of 256, 0.49 with 36-byte records moved through
// memory and back in input order. 1024 pp events of 60 tracks: 0.044 ms in CTAs of 64 threads, 0.24 in
// CTAs of 512.
constexpr size_t sort_shared_bytes(int warps)
{
  return sizeof(int) * ((size_t)warps * kBuckets + 3 * kBuckets + 34 + 4 + (size_t)warps * 32 * kClusterWords);
}

template <int kThreads_>
__global__ void __launch_bounds__(kThreads_, 1536 / kThreads_) k_cluster_sort(Arena a)
{
  constexpr int kWarps = kThreads_ / 32;
  namespace cg = cooperative_groups;
  extern __shared__ int shared[];
  int *const hist_all = shared;  // [kWarps][kBuckets]
  int *const cta_total = hist_all + kWarps * kBuckets;
  int *const bucket_total = cta_total + kBuckets;
  int *const bucket_base = bucket_total + kBuckets;
  int *const scan_totals = bucket_base + kBuckets;  // [33]
  int *const s_flags = scan_totals + 34;            // irregular, least r, largest r (float bits)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ctas = (int)cg::this_cluster().num_blocks(), rank = (int)cg::this_cluster().block_rank();
  const int seg = blockIdx.x / ctas;
  const int e = seg / ITSU_LAYERS, layer = seg % ITSU_LAYERS;
  const int64_t begin = a.layer_off[seg];
  const int n = (int)(a.layer_off[seg + 1] - begin);
  const int64_t raw_begin = a.raw_off ? a.raw_off[seg] : begin;  // frames share raw clusters
  const float vx = a.vtx[3 * e], vy = a.vtx[3 * e + 1], vz = a.vtx[3 * e + 2];
  int *const hist = hist_all + warp * kBuckets;
  int32_t *const stage = s_flags + 4 + warp * 32 * kClusterWords;

  // by input index: bucket; by sorted position: input index (perm)
  uint32_t *const perm = a.sort_index + begin;
  uint32_t *const bucket = perm + a.sort_stride;
  auto sync_segment = [&]() {
    if (ctas == 1) {
      __syncthreads();
    } else {
      cg::this_cluster().sync();
    }
  };

  if (tid == 0 && layer == 0 && rank == 0) {
    const bool ok = isfinite(vx) && isfinite(vy) && isfinite(vz) && fabsf(vx) <= kMaxAbsCoordinate &&
                    fabsf(vy) <= kMaxAbsCoordinate && fabsf(vz) <= kMaxAbsCoordinate;
    if (!ok) {
      atomicOr(&a.status->flags, kFlagInvalid);
      atomicMin(&a.status->invalid_event, e);
    }
  }
  for (int k = tid; k < kWarps * kBuckets; k += kThreads_) {
    hist_all[k] = 0;
  }
  if (tid == 0) {
    s_flags[0] = 0;
    s_flags[1] = 0x7f800000;
    s_flags[2] = 0;
  }
  __syncthreads();

  // Pass 1: transform every cluster (input order), per-warp bucket histograms. Each warp owns a
  // consecutive input range and moves it through its stage 32 clusters at a time.
  const int chunk = (n + ctas * kWarps - 1) / (ctas * kWarps);
  const int wb = min(n, (rank * kWarps + warp) * chunk), we = min(n, wb + chunk);
  float4 *const recs = a.sort_recs + 2 * begin;
  unsigned irregular = 0, rmin = 0x7f800000u, rmax = 0;  // of r's float bits: r >= 0 orders like its bits
  for (int i0 = wb; i0 < we; i0 += 32) {
    const int count = min(32, we - i0);
    itsu_cluster c{};
    if (a.raw_track) {
      // 16-byte input records (x, y, z, MC id): one aligned 16-byte load per lane; the cluster id
      // is the record's index in its layer's input order, alpha 0
      if (lane < count) {
        const float4 q = reinterpret_cast<const float4 *>(a.raw_track + raw_begin + i0)[lane];
        c.x = q.x;
        c.y = q.y;
        c.z = q.z;
        c.cluster_id = i0 + lane;
        c.alpha = 0.0f;
        c.mc_id = __float_as_int(q.w);
      }
    } else {
      __syncwarp();  // the stage is refilled
      if (a.raw_in) {
        stage_in_words<kClusterInWords>(stage, a.raw_in + raw_begin + i0, count);
        if (lane < count) {
          c = stage_get_in(stage, lane);
        }
      } else {
        stage_in(stage, a.raw + raw_begin + i0, count);
        if (lane < count) {
          c = stage_get(stage, lane);
        }
      }
    }
    if (lane < count) {
      const int i = i0 + lane;
      const Transformed t = transform_cluster(layer, c.x, c.y, c.z, vx, vy);
      const bool ok = isfinite(c.x) && isfinite(c.y) && isfinite(c.z) && fabsf(c.x) <= kMaxAbsCoordinate &&
                      fabsf(c.y) <= kMaxAbsCoordinate && fabsf(c.z) <= kMaxAbsCoordinate && !(t.r == 0.0f && c.z == vz);
      if (!ok) {
        atomicOr(&a.status->flags, kFlagInvalid);
        atomicMin(&a.status->invalid_index, (int)(begin + i));
      }
      recs[2 * i] = make_float4(c.x, c.y, c.z, t.r);
      recs[2 * i + 1] = make_float4(t.phi, __int_as_float(c.cluster_id), c.alpha, __int_as_float(c.mc_id));
      const int zb = z_bin_index(layer, c.z), pb = phi_bin_index(t.phi);
      irregular |= zb < 0 || zb >= kZBins || pb < 0 || pb >= kPhiBins;
      rmin = min(rmin, __float_as_uint(t.r));
      rmax = max(rmax, __float_as_uint(t.r));
      const int b = bucket_of(t.bin);
      bucket[i] = (uint32_t)b;
      atomicAdd(&hist[b], 1);
    }
  }
  irregular = __reduce_or_sync(0xffffffffu, irregular);
  rmin = __reduce_min_sync(0xffffffffu, rmin);
  rmax = __reduce_max_sync(0xffffffffu, rmax);
  if (lane == 0) {
    atomicOr(&s_flags[0], (int)irregular);
    atomicMin(&s_flags[1], (int)rmin);
    atomicMax(&s_flags[2], (int)rmax);
  }
  __syncthreads();

  // Pass 2: per-bucket prefix over warps (and CTAs), exclusive scan over buckets, index table.
  for (int b = tid; b < kBuckets; b += kThreads_) {
    int s = 0;
    for (int w = 0; w < kWarps; ++w) {
      const int v = hist_all[w * kBuckets + b];
      hist_all[w * kBuckets + b] = s;
      s += v;
    }
    cta_total[b] = s;
    bucket_total[b] = s;
  }
  sync_segment();
  int seg_irregular = s_flags[0], seg_rmin = s_flags[1], seg_rmax = s_flags[2];
  if (ctas > 1) {
    for (int c = 0; c < ctas; ++c) {
      const int *other = cg::this_cluster().map_shared_rank(s_flags, c);
      seg_irregular |= other[0];
      seg_rmin = min(seg_rmin, other[1]);
      seg_rmax = max(seg_rmax, other[2]);
    }
    for (int b = tid; b < kBuckets; b += kThreads_) {
      int before = 0, all = 0;
      for (int c = 0; c < ctas; ++c) {
        const int v = cg::this_cluster().map_shared_rank(cta_total, c)[b];
        before += c < rank ? v : 0;
        all += v;
      }
      bucket_total[b] = all;
      for (int w = 0; w < kWarps; ++w) {
        hist_all[w * kBuckets + b] += before;
      }
    }
    __syncthreads();
  }
  for (int b0 = 0, carry = 0; b0 < kBuckets; b0 += kThreads_) {
    const int b = b0 + tid;
    const int v = b < kBuckets ? bucket_total[b] : 0;
    int total;
    const int ex = block_exclusive_scan<int>(v, scan_totals, total);
    if (b < kBuckets) {
      bucket_base[b] = carry + ex;
    }
    carry += total;
  }
  __syncthreads();
  if (layer > 0) {
    // table[b] = first sorted index with bin >= b = #clusters with bin < b for b >= 1; table[0] = 0
    // (PrimaryVertexContext.cxx:90-119: negative bins never move the fill cursor off bin 0).
    int32_t *table = a.index_tables + ((int64_t)e * ITSU_TRACKLET_LAYERS + layer - 1) * kTableSize;
    for (int b = rank * kThreads_ + tid; b < kTableSize; b += ctas * kThreads_) {
      table[b] = b == 0 ? 0 : bucket_base[b + 1];
    }
  }

  // Pass 3: each cluster's sorted position. Warps own consecutive input ranges whose bucket offsets
  // were prefixed in warp order; inside a warp, lanes of equal bucket rank by lane order.
  for (int i0 = wb; i0 < we; i0 += 32) {
    const int i = i0 + lane;
    const bool valid = i < we;
    const int b = valid ? (int)bucket[i] : -1 - lane;
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    const int before = __popc(peers & ((1u << lane) - 1u));
    int pos = 0;
    if (valid) {
      pos = bucket_base[b] + hist[b] + before;
      perm[pos] = (uint32_t)i;
    }
    __syncwarp();
    if (valid && (peers >> lane) == 1u) {  // the highest lane of its bucket
      hist[b] += before + 1;
    }
    __syncwarp();
  }
  sync_segment();

  // Negative bins share bucket 0 in input order; order them by bin, stably. A bottom-up merge sort of
  // (bin, input index) between two pairs of arrays: in each
  // round, runs of `width` are merged in pairs, every cluster moving to (its place in its run) + (the
  // clusters of the partner run that go before it: smaller bins, and for the right run equal bins
  // too), so ties keep input order. O(m log^2 m) work, for layers with many clusters beyond the z range.
  const int m = bucket_total[0];
  if (m > 1) {
    if (rank == 0) {
      int *key = reinterpret_cast<int *>(bucket + a.sort_stride), *key_to = key + a.sort_stride;
      uint32_t *idx = perm, *idx_to = bucket;
      for (int i = tid; i < m; i += kThreads_) {
        const int from = (int)perm[i];
        key[i] = bin_index(z_bin_index(layer, recs[2 * from].z), phi_bin_index(recs[2 * from + 1].x));
      }
      for (int width = 1; width < m; width *= 2) {
        __syncthreads();
        for (int i = tid; i < m; i += kThreads_) {
          const int run = i / width;
          const bool left = (run & 1) == 0;
          const int own_start = run * width;
          const int other_start = left ? own_start + width : own_start - width;
          const int other_end = min(other_start + width, m);
          const int k = key[i];
          int lo = other_start, hi = max(other_start, other_end);  // an empty partner run: no move
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key[mid] < k || (!left && key[mid] == k)) {
              lo = mid + 1;
            } else {
              hi = mid;
            }
          }
          const int to = min(own_start, other_start) + (i - own_start) + (lo - other_start);
          key_to[to] = k;
          idx_to[to] = idx[i];
        }
        int *const t = key;
        key = key_to;
        key_to = t;
        uint32_t *const u = idx;
        idx = idx_to;
        idx_to = u;
      }
      __syncthreads();
      if (idx != perm) {
        for (int i = tid; i < m; i += kThreads_) {
          perm[i] = idx[i];
        }
      }
    }
    sync_segment();
  }

  // What lets the tracklet stage prune: a layer is regular when every cluster has a z bin and a phi bin
  // inside the 20 x 20 table (then a bin's column is its clusters' z bin). Its r range stands beside.
  // (Layer 0 is never the outer layer of a tracklet.)
  if (a.clu_key != nullptr && layer > 0 && rank == 0 && tid == 0) {
    a.seg_regular[seg] = !seg_irregular && m == 0 && bucket_total[kBuckets - 1] == 0;
    a.seg_rrange[seg] = make_float2(__int_as_float(seg_rmin), __int_as_float(seg_rmax));
  }
  // Pass 4: every output in sorted order.
  for (int i0 = (rank * kWarps + warp) * 32; i0 < n; i0 += ctas * kThreads_) {
    const int count = min(32, n - i0);
    __syncwarp();  // the stage is refilled
    if (lane < count) {
      const int pos = i0 + lane;
      const int64_t at = begin + pos;
      const int i = (int)perm[pos];
      const float4 p = recs[2 * i], q = recs[2 * i + 1];
      itsu_cluster c;
      c.x = p.x;
      c.y = p.y;
      c.z = p.z;
      c.phi = q.x;
      c.r = p.w;
      c.cluster_id = __float_as_int(q.y);
      c.alpha = q.z;
      c.mc_id = __float_as_int(q.w);
      c.bin = bin_index(z_bin_index(layer, c.z), phi_bin_index(c.phi));
      stage_put(stage, lane, c);
      if (a.xyzr) {
        a.xyzr[at] = p;
        a.phi[at] = c.phi;
        a.clu_aux[at] = make_int4(c.cluster_id, __float_as_int(c.alpha), c.mc_id, c.bin);
        a.clu_seg[at] = seg;
        a.clu_key[at] = cluster_key(layer, c.z, c.phi);
      }
    }
    stage_out(a.sorted + begin + i0, stage, count);
  }
}

// ------------------------------------------------------------------------------------------
// (b) tracklets: TrackerTraits<false>::computeLayerTracklets (Tracker.cxx:45-117)

// Tracklet layer L of event e runs only if every layer pair up to L has clusters (:49-52).
__device__ __forceinline__ bool tracklets_active(const int32_t *lo, int layer)
{
  for (int l = 0; l <= layer; ++l) {
    if (lo[l + 1] - lo[l] <= 0 || lo[l + 2] - lo[l + 1] <= 0) {
      return false;
    }
  }
  return true;
}

// Tracklet.cxx:32-40: the tracklet from inner cluster c to outer cluster d (local indices given);
// write_tracklet stores the one from flat cluster i_flat to j_flat.
__device__ __forceinline__ itsu_tracklet make_tracklet(float4 c, float4 d, int32_t c_local, int32_t d_local)
{
  itsu_tracklet t;
  t.first_cluster = c_local;
  t.second_cluster = d_local;
  t.tan_lambda = (c.z - d.z) / (c.w - d.w);
  t.phi = itsu_atan2f(c.y - d.y, c.x - d.x);
  return t;
}

// The record in one 16-byte store (the struct's own alignment of 4 would make it four), and its key.
__device__ __forceinline__ void store_tracklet(const Arena &a, int64_t out, const itsu_tracklet &t)
{
  reinterpret_cast<int4 *>(a.tracklets)[out] =
      make_int4(t.first_cluster, t.second_cluster, __float_as_int(t.tan_lambda), __float_as_int(t.phi));
  a.trk_key[out] = tracklet_key(t.tan_lambda, t.phi);
}

__device__ __forceinline__ itsu_tracklet load_tracklet(const Arena &a, int64_t k)
{
  const int4 w = reinterpret_cast<const int4 *>(a.tracklets)[k];
  itsu_tracklet t;
  t.first_cluster = w.x;
  t.second_cluster = w.y;
  t.tan_lambda = __int_as_float(w.z);
  t.phi = __int_as_float(w.w);
  return t;
}

__device__ __forceinline__ void write_tracklet(const Arena &a, int out, int64_t i_flat, int64_t j_flat, int seg)
{
  store_tracklet(a, out, make_tracklet(a.xyzr[i_flat], a.xyzr[j_flat], (int32_t)(i_flat - a.layer_off[seg]),
                                       (int32_t)(j_flat - a.layer_off[seg + 1])));
  if (out % 32 == 0) {
    a.trk_seg32[out / 32] = seg - seg / ITSU_LAYERS;  // 7 e + L to 6 e + L
  }
}

constexpr int kTrackletSlots = kTrackletSlotsPerCluster;
constexpr int kMaskKeys = 32;  // keys of the walk's window a mask holds (with 64 the pass took 0.72 ms per 128 central events when with 32 it took 0.66; it takes 0.59 now)
constexpr int kMaxMaskedOut = 64;  // out-degrees up to this are evaluated pair-parallel with a pass mask

// The reference's candidate sequence of one inner cluster (Tracker.cxx:73-113), calling
// on_pass(j) for every next-layer cluster j that passes the cut, in emission order: the phi
// rows of the bin window in wrap-around order and, in each row, the sorted clusters from the
// row's first bin through the first cluster at or after the window's end (inclusive bound, with
// the P1/P5 guards).
//
// On a regular next layer the row is pruned, which is exact: a pass needs |P - z2| < dz with
// P = (tanL (r2 - r1) + z1) in binary32, P is monotone in r2, so every passing z2 lies within
// [P(rmin) - dz, P(rmax) + dz] (widened by 1e-3 cm for the rounding of the bounds); only the z bins of
// the row that meet that interval can hold passes, and of their clusters (consecutive ones) those
// whose 4-byte keys lie in the window (TrackletWindow, a superset of the cut) are tested. The row's
// last candidate (the inclusive bound, past the window's z bins) is always evaluated. Irregular layers
// take the reference walk.
struct TrackletProbe {
  float4 c;      // inner cluster (x, y, z, r)
  float phi1, tan_lambda, max_dz;
  const float4 *xyzr;  // next layer
  const float *phi;
  GateWindow win;      // kGate: the learned form's first-stage windows

  // Tracker.cxx:93-100 for a next-layer cluster at z2, r2, phi2; kGate: and inside the windows
  template <bool kGate>
  __device__ __forceinline__ bool pass(float z2, float r2, float phi2) const
  {
    const float delta_z = fabsf(tan_lambda * (r2 - c.w) + c.z - z2);
    const float delta_phi = fabsf(phi1 - phi2);
    const bool cut = delta_z < max_dz && (delta_phi < kPhiCoordinateCut || delta_phi > kPhiWrapTracklet);
    if constexpr (kGate) {
      return cut && gate_window_pass(win, make_float4(0.0f, 0.0f, z2, r2), phi2);
    }
    return cut;
  }

  template <bool kGate>
  __device__ __forceinline__ bool pass(int j) const
  {
    const float2 d = reinterpret_cast<const float2 *>(xyzr + j)[1];  // z, r
    return pass<kGate>(d.x, d.y, phi[j]);
  }
};

// The walk state of one inner cluster i (flat index): whether its layer runs the tracklet
// stage, and the probe, window and pruning bounds of its candidate walk.
struct InnerCluster {
  bool walk;
  int win_row, win_rows;  // the phi rows its |dphi| window reaches (win_rows = kPhiBins: every row)
  int seg, e, layer;
  int4 rect;
  TrackletProbe probe;
  bool prune;
  int zb_lo, zb_hi, zb_top;  // the z bins walked of a row; clusters of bins above zb_top have z beyond the cut
  KeyWindow window;
  const int32_t *table;
  int n_next;
  int64_t next_begin;
};

// The phi rows that hold the azimuths within half_width of phi (the window's rows, clamped into
// 0..kPhiBins - 1): first row and count, in the walk's cyclic order.
__device__ __forceinline__ void window_rows(float phi, float half_width, int *first, int *rows)
{
  float lo = phi - half_width, hi = phi + half_width;
  lo = lo < 0.0f ? lo + kTwoPi : lo;
  hi = hi >= kTwoPi ? hi - kTwoPi : hi;
  const int r_lo = min(phi_bin_index(lo), kPhiBins - 1), r_hi = min(phi_bin_index(hi), kPhiBins - 1);
  int n = r_hi - r_lo + 1;
  *first = r_lo;
  *rows = n <= 0 ? n + kPhiBins : n;
}

// With a tracklet gate (learned form), its first stage's windows for the layer narrow the walk: a
// tracklet outside them is not kept. The walk keeps the plain rect and its row sequence (with the
// reference's edge behaviour, e.g. a first row of 20 when the window's lower edge rounds to 2pi),
// but of a row outside the |dphi| window (widened by 1e-3 rad against rounding) it only tests the
// row's bound candidate (P1), which can lie in the next row; the pruned columns take the narrower
// z range of the |dz| window (widened by 1e-3 cm). In a regular layer every cluster sits in its
// own bin, so the walk still meets every plain candidate inside the windows, in the plain order;
// other layers are walked whole. Every candidate's cut includes the windows themselves
// (gate_window_pass): the gated tracklets are exactly the plain tracklets inside the windows.
// kGate: the learned form with a tracklet gate (a.gate set); the plain form's instantiation has
// none of the windows' code.
template <bool kGate>
__device__ __forceinline__ InnerCluster inner_cluster(const Arena &a, int64_t i)
{
  InnerCluster s;
  s.walk = false;
  s.seg = a.clu_seg[i];
  s.e = s.seg / ITSU_LAYERS;
  s.layer = s.seg % ITSU_LAYERS;
  const int32_t *lo = a.layer_off + s.e * ITSU_LAYERS;
  if (s.layer >= ITSU_LAYERS - 1 || !tracklets_active(lo, s.layer)) {
    return s;
  }
  s.probe.c = a.xyzr[i];
  s.probe.phi1 = a.phi[i];
  const float vz = a.vtx[3 * s.e + 2];
  s.probe.tan_lambda = (s.probe.c.z - vz) / s.probe.c.w;
  const float dir_z = s.probe.tan_lambda * (kC.r[s.layer + 1] - s.probe.c.w) + s.probe.c.z;
  s.rect = bins_rect(s.probe.phi1, s.layer, dir_z);
  if (s.rect.x == 0 && s.rect.y == 0 && s.rect.z == 0 && s.rect.w == 0) {
    return s;  // the reference's "no bins" rect (Tracker.cxx:66-70)
  }
  s.walk = true;
  s.next_begin = lo[s.layer + 1];
  s.probe.xyzr = a.xyzr + s.next_begin;
  s.probe.phi = a.phi + s.next_begin;
  s.probe.max_dz = kC.trk_max_dz[s.layer];
  const int next_seg = s.seg + 1;
  const bool regular = a.prune_tracklets != 0 && a.seg_regular[next_seg] != 0;
  s.win_row = 0;
  s.win_rows = kPhiBins;
  float half = s.probe.max_dz, reach = kPhiCoordinateCut;
  if constexpr (kGate) {
    s.probe.win = gate_window(*a.gate, s.layer, s.probe.c, s.probe.phi1, vz);
    if (regular && s.probe.win.dphi + 1e-3f < kPhiCoordinateCut) {  // a wider window narrows nothing
      reach = s.probe.win.dphi + 1e-3f;
      window_rows(s.probe.phi1, reach, &s.win_row, &s.win_rows);
    }
    half = fminf(half, s.probe.win.dz + 1e-3f);
  }
  s.prune = regular;
  if (regular) {
    const float2 rr = a.seg_rrange[next_seg];
    const float p1 = s.probe.tan_lambda * (rr.x - s.probe.c.w) + s.probe.c.z;
    const float p2 = s.probe.tan_lambda * (rr.y - s.probe.c.w) + s.probe.c.z;
    const float zlo = fminf(p1, p2) - half - 1e-3f, zhi = fmaxf(p1, p2) + half + 1e-3f;
    s.prune = isfinite(zlo) && isfinite(zhi);
    s.zb_lo = max(s.rect.x, z_bin_index(s.layer + 1, zlo));
    s.zb_top = z_bin_index(s.layer + 1, zhi);
    s.zb_hi = min(s.rect.z, s.zb_top);
    s.window = tracklet_window(s.layer + 1, s.probe.phi1, reach, zlo, zhi);
  }
  s.table = a.index_tables + ((int64_t)s.e * ITSU_TRACKLET_LAYERS + s.layer) * kTableSize;
  s.n_next = lo[s.layer + 2] - lo[s.layer + 1];
  return s;
}

// win_row, win_rows: the phi rows whose candidates are walked (win_rows = kPhiBins: every row); of
// the other rows only the bound candidate is tested (the first cluster of the first bin after the
// row's last z column: past empty bins it can lie in any later row).
template <bool kGate, typename OnPass>
__device__ __forceinline__ void walk_inner(const Arena &a, const InnerCluster &s, OnPass &&on_pass)
{
  const int4 rect = s.rect;
  int phi_bins = rect.w - rect.y + 1;
  if (phi_bins < 0) {
    phi_bins += kPhiBins;
  }
  for (int phi_bin = rect.y, phi_count = 0; phi_count < phi_bins;
       phi_bin = (phi_bin + 1 == kPhiBins) ? 0 : phi_bin + 1, ++phi_count) {
    const int first_bin = bin_index(rect.x, phi_bin);
    const int max_bin = min(first_bin + rect.z - rect.x + 1, kTableBins);  // P5
    const bool walk_row = s.win_rows >= kPhiBins ||
                          (phi_bin < kPhiBins && (phi_bin - s.win_row + kPhiBins) % kPhiBins < s.win_rows);
    if (s.prune && phi_bin < kPhiBins) {
      if (walk_row && s.zb_lo <= s.zb_hi) {
        const int k0 = s.table[phi_bin * kZBins + s.zb_lo], k1 = s.table[phi_bin * kZBins + s.zb_hi + 1];
        // the keys in aligned groups of four (the array has room for the last group's overrun), a mask
        // of kMaskKeys at a time
        const int skip = (int)((s.next_begin + k0) & 3);
        const uint4 *keys = reinterpret_cast<const uint4 *>(a.clu_key + (s.next_begin + k0 - skip));
        for (int at = k0 - skip; at < k1; at += kMaskKeys, keys += kMaskKeys / 4) {
          const int n = min(kMaskKeys, k1 - at);
          // (the compiler's own unrolling: of 1, 2, 4 and 8 it is slower, 0.65 to 0.76 ms per 128 central events)
          uint32_t mask = 0;
          for (int b = 0; b < n; b += 4) {
            mask |= key_window_four(s.window, keys[b / 4]) << b;
          }
          if (at < k0) {
            mask &= ~0u << skip;
          }
          mask &= ~0u >> (kMaskKeys - n);
          while (mask) {
            const int j = at + __ffs((int)mask) - 1;
            mask &= mask - 1;
            if (s.probe.template pass<kGate>(j)) {
              on_pass(j);
            }
          }
        }
      }
      // The inclusive bound's candidate (P1: inside the layer): the first cluster of bin
      // max_bin, the row's next z column. When that bin is not empty and its z column lies
      // beyond zhi's (z bins are monotone in z; a regular layer's clusters sit in exactly their
      // bins), the candidate's z exceeds zhi and it fails the dz cut: it is not read.
      const int x = s.table[max_bin];
      const bool beyond = rect.z + 1 < kZBins && rect.z + 1 > s.zb_top && s.table[max_bin + 1] > x;
      if (!beyond && x < s.n_next && s.probe.template pass<kGate>(x)) {
        on_pass(x);
      }
    } else {
      const int first_row = s.table[first_bin];
      const int last_row = min(s.table[max_bin], s.n_next - 1);  // inclusive bound, P1
      for (int j = walk_row ? first_row : last_row; j <= last_row; ++j) {
        if (s.probe.template pass<kGate>(j) && (walk_row || j == s.table[max_bin])) {
          on_pass(j);
        }
      }
    }
  }
}

constexpr int kCountThreads = 256;

// Count pass, one thread per inner cluster: the number of tracklets, and the outer clusters of
// the first kTrackletSlots of them in emission order. kGate: the learned form's first stage
// (inner_cluster). At most kCountThreads threads per block. Bound by the integer pipe, half of whose
// work is lost to lanes whose candidates end at different times: 0.59 ms per 128 central events (0.63
// at five blocks per SM); with a walk of z-sorted lists (a binary search per bin and passes put back
// into index order) 0.62, and 0.09 ms more in the clustering; with the candidates of all lanes queued
// and the cut in full rounds 0.74.
template <bool kGate>
__global__ void __launch_bounds__(kCountThreads, kGate ? 5 : 6) k_tracklets_count(Arena a)
{
  const int64_t i = global_thread();
  const bool valid = i < a.n_clusters;
  int count = 0;
  InnerCluster s;
  s.walk = false;
  if (valid) {
    s = inner_cluster<kGate>(a, i);
  }
  if (s.walk) {
    walk_inner<kGate>(a, s, [&](int j) {
      if (count < kTrackletSlots) {
        a.trk_slots[count * a.slot_stride + i] = j;
      }
      ++count;
    });
  }
  // the warp's 32 clusters lie in one scan tile: their tracklets go to its sum
  const unsigned long long warp_count = warp_sum(0xffffffffu, (unsigned)count);
  if ((threadIdx.x & 31) == 0 && warp_count != 0) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&a.scan_partials[i / kScanTile]), warp_count);
  }
  if (!valid) {
    return;
  }
  a.trk_count[i] = count;
  if (count > kTrackletSlots) {  // rare: the write pass leaves this cluster to k_tracklets_crowded
    const unsigned long long q = atomicAdd(reinterpret_cast<unsigned long long *>(&a.status->trk_crowded), 1ull);
    if ((int64_t)q < a.n_clusters) {
      a.clu_crowded[q] = (int32_t)i;
    }
  }
}

template <typename T>
__device__ __forceinline__ T warp_exclusive_sum(T v, T &total)
{
  const int lane = threadIdx.x & 31;
  T inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) {
      inc += t;
    }
  }
  total = __shfl_sync(0xffffffffu, inc, 31);
  return inc - v;
}

// Owner lane of flattened item t given the lanes' exclusive prefix sums: the last lane whose
// prefix is <= t (for t < total this lane holds item t). All lanes must call it together.
template <typename T>
__device__ __forceinline__ int owner_of(T excl, T t)
{
  int owner = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    const T v = __shfl_sync(0xffffffffu, excl, owner + step);
    if (v <= t) {
      owner += step;
    }
  }
  return owner;
}

// Learned form: the tracklet gate. After the count pass and before the tracklet scan, a warp per
// 32 consecutive inner clusters scores their tracklets (the outer clusters the count pass kept in
// their slots), 32 at a time on the tensor cores (8 -> 16 -> 16 -> 1, ReLU, BF16 / FP32, the
// network in registers), keeps those whose logit is not below the gate's threshold (a NaN logit
// keeps its tracklet), moves the kept slots to the front in their order and lowers the cluster's
// count and its scan tile's sum by the dropped ones. The write pass then writes the kept tracklets
// in emission order, as in the plain form. Inner clusters with more than kTrackletSlots tracklets
// keep all of them, unscored (the crowded pass writes them), and so do those of the layers the
// network does not score (the model's mlp_layers).
//
// Per warp and group of 32 clusters, the flattened tracklets' owners and ranks are listed once in
// shared memory (each cluster's lane writes its own entries), and each cluster's gate state (what
// its features need of it) sits beside them, so that a tile reads its rows' owners, states and
// slots without searches or shuffles; the lanes holding a row's logit keep or drop it.
constexpr int kGateThreads = 256;
constexpr int kGateWarps = kGateThreads / 32;

struct __align__(16) GateLane {
  GateInner g;
  int32_t next;  // first cluster of the next layer
  int32_t pad_;
};

// The gate pass's per-warp shared memory.
struct GateShared {
  __align__(16) __nv_bfloat16 rows[kGateWarps][32][kMlpIn];
  unsigned long long keep[kGateWarps][32];
  uint16_t owner_rank[kGateWarps][32 * kTrackletSlots];  // owner lane * 64 + rank
  GateLane lanes[kGateWarps][32];
};

// One warp group of k_tracklets_gate: the inner clusters base .. base + 31 of which those in
// [start, end) take part (event e).
__device__ __forceinline__ void gate_group(const Arena &a, const GateSmem &net, const GateRegs &R, GateShared &sh, int warp,
                                           int64_t base, int64_t start, int64_t end, int e)
{
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  __nv_bfloat16 (&rows)[32][kMlpIn] = sh.rows[warp];
  unsigned long long (&keep)[32] = sh.keep[warp];
  uint16_t (&owner_rank)[32 * kTrackletSlots] = sh.owner_rank[warp];
  GateLane (&lanes)[32] = sh.lanes[warp];
  const int64_t i = base + lane;
  int count = 0;
  bool scored = false;  // by the network: in the range, and not crowded
  if (i >= start && i < end) {
    count = a.trk_count[i];
    if (count > 0 && count <= kTrackletSlots) {
      const int seg = a.clu_seg[i];
      scored = true;
      GateLane &s = lanes[lane];
      s.g = gate_inner(seg % ITSU_LAYERS, a.xyzr[i], a.phi[i], a.vtx[3 * e], a.vtx[3 * e + 1], a.vtx[3 * e + 2]);
      s.next = a.layer_off[seg + 1];
    }
  }
  const int mine = scored ? count : 0;
  keep[lane] = 0ull;
  int total = 0;
  const int excl = warp_exclusive_sum(mine, total);
  for (int r = 0; r < mine; ++r) {
    owner_rank[excl + r] = (uint16_t)(lane * 64 + r);
  }
  __syncwarp();
  for (int p0 = 0; p0 < total; p0 += 32) {
    const int p = p0 + lane;
    float f[kMlpIn];
    if (p < total) {
      const int orank = owner_rank[p], owner = orank >> 6, rank = orank & 63;
      const GateLane &o = lanes[owner];
      const int64_t j = o.next + a.trk_slots[(int64_t)rank * a.slot_stride + base + owner];
      gate_features(o.g, a.xyzr[j], a.phi[j], f);
    } else {
#pragma unroll
      for (int k = 0; k < kMlpIn; ++k) {
        f[k] = net.mean[k];
      }
    }
    *reinterpret_cast<uint4 *>(&rows[lane][0]) = gate_row(net.mean, net.inv_std, f);
    __syncwarp();
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      float lo, hi;
      gate_forward_m16(R, rows, mt, lo, hi);
      if (t == 0) {  // this lane holds the logits of rows 16 mt + g and 16 mt + g + 8
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = p0 + mt * 16 + g + 8 * h;
          const float logit = h ? hi : lo;
          if (q < total && !(logit < net.threshold)) {
            const int orank = owner_rank[q];
            atomicOr(&keep[orank >> 6], 1ull << (orank & 63));
          }
        }
      }
    }
    __syncwarp();  // the rows are refilled for the next tile
  }
  // kept slots to the front, in order (coalesced across the warp's clusters, slot by slot)
  const unsigned long long m = keep[lane];
  const int scan_to = __reduce_max_sync(0xffffffffu, (unsigned)mine);
  int kept = 0;
  for (int q = 0; q < scan_to; ++q) {
    if (q < count && ((m >> q) & 1ull)) {
      if (kept != q) {
        a.trk_slots[(int64_t)kept * a.slot_stride + i] = a.trk_slots[(int64_t)q * a.slot_stride + i];
      }
      ++kept;
    }
  }
  int dropped = 0;
  if (scored) {
    a.trk_count[i] = kept;
    dropped = count - kept;
  }
  // the warp's 32 clusters lie in one scan tile (the count pass added their tracklets to its sum)
  const int warp_dropped = (int)__reduce_add_sync(0xffffffffu, (unsigned)dropped);
  if (lane == 0 && warp_dropped != 0) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&a.scan_partials[base / kScanTile]),
              (unsigned long long)(-(int64_t)warp_dropped));
  }
  __syncwarp();
}

__global__ void __launch_bounds__(kGateThreads) k_tracklets_gate(Arena a)
{
  __shared__ GateSmem net;
  __shared__ GateShared sh;
  load_mlp(net, *a.gate);
  __syncthreads();
  const GateRegs R = gate_regs(net);
  const int warp = threadIdx.x >> 5;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t first_warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  for (int e = blockIdx.y; e < a.n_events; e += gridDim.y) {
    for (int l0 = 0; l0 < ITSU_TRACKLET_LAYERS; ++l0) {
      if (!((net.layers >> l0) & 1u) || (l0 > 0 && ((net.layers >> (l0 - 1)) & 1u))) {
        continue;  // not the first layer of a run of scored layers
      }
      int l1 = l0;
      while (l1 + 1 < ITSU_TRACKLET_LAYERS && ((net.layers >> (l1 + 1)) & 1u)) {
        ++l1;
      }
      // the inner clusters of layers l0..l1 of event e, in warp groups aligned to 32 (so that each
      // group lies in one scan tile; a group's lanes outside the range take no part)
      const int64_t start = a.layer_off[e * ITSU_LAYERS + l0], end = a.layer_off[e * ITSU_LAYERS + l1 + 1];
      for (int64_t base = (start & ~(int64_t)31) + first_warp * 32; base < end; base += warps * 32) {
        gate_group(a, net, R, sh, warp, base, start, end, e);
      }
    }
  }
}

// Write pass, a warp per 32 consecutive inner clusters: the warp's lanes fill their clusters' tracklets
// together, each taking the next one: it finds its inner cluster (owner) and rank there, reads the
// outer cluster the count pass kept in that slot, and writes the tracklet (Tracklet.cxx:32-40) and its
// key with coalesced stores; all lanes compute their binary64 azimuths together. What a
// tracklet needs of its owner stands in shared memory. Each cluster's tracklets lookup entry is
// written here too, and the segment of every 32nd tracklet. The tracklets of an inner cluster with
// more than kTrackletSlots of them (not kept by the count pass) come from write_crowded.
// Runs over the inner clusters [c0, c1) (c0 a multiple of 32, so that warps hold whole aligned
// groups of 32 clusters): all of them, or one event group's share of them.
// Bound by the slots' and outer clusters' gathers with the azimuth's issue: 0.475 ms per 128 central
// events (0.488 with a segment id per tracklet; the figures below before the prefetch): 0.50 at five blocks per SM (48 registers), 0.55 at six (the slots' lines, which a warp comes back
// to, leave L1 too soon) or four; 0.58 with the owners' values in shuffles, the correctly rounded
// division and the azimuth's double-double path inlined. Slots of a cluster side by side: 0.56.
constexpr int kWriteThreads = 256;
constexpr int kWriteBlocks = 5;  // resident blocks per SM
// A block prefetches the lines of the block a wave later: coordinates, offsets, segments and the first
// slots (0.499 ms without; 12 slots and 16 cost more than they bring, 0.490 and 0.496, two waves 0.509).
constexpr int kWriteAhead = 148 * kWriteBlocks;  // of the 148 SMs of a B200
constexpr int kWriteAheadSlots = 8;
static_assert(kWriteAheadSlots <= kTrackletSlots && 6 + kWriteAheadSlots <= 32, "a line per lane");

struct WriteWarp {
  float4 c[32];
  int4 owner[32];  // first tracklet less the lanes' prefix, the prefix, cluster in its layer, first cluster of the next layer
  int32_t sid[32];
};

__global__ void __launch_bounds__(kWriteThreads, kWriteBlocks) k_tracklets_write(Arena a, int64_t c0, int64_t c1)
{
  __shared__ WriteWarp shared[kWriteThreads / 32];
  // not stopped by the scratch flag: with event groups the count pass of an earlier group may have raised
  // it, and this group's goes on to add up what the run needs, on tracklets that have to be there
  if ((*(volatile const int32_t *)&a.status->flags & kCapacityMask & ~kFlagCapScratch) != 0) {
    return;
  }
  WriteWarp &w = shared[threadIdx.x >> 5];
  const int64_t i = c0 + global_thread();
  const int lane = threadIdx.x & 31;
  {
    const int64_t next = i - lane + (int64_t)kWriteAhead * kWriteThreads;
    if (next + 32 <= c1) {
      const void *line = lane < 4 ? (const void *)(a.xyzr + next + lane * 8)
                                  : (lane == 4 ? (const void *)(a.trk_off + next)
                                               : (lane == 5 ? (const void *)(a.clu_seg + next)
                                                            : (const void *)(a.trk_slots + (lane - 6) * a.slot_stride + next)));
      if (lane < 6 + kWriteAheadSlots) {
        prefetch_line(line);
      }
    }
  }
  int32_t first = 0, count = 0;
  int seg = 0, sid = 0;
  if (i < c1) {
    first = a.trk_off[i];
    count = a.trk_off[i + 1] - first;
    a.trk_range[i] = make_int2(first, count);
    seg = a.clu_seg[i];
    const int e = seg / ITSU_LAYERS, layer = seg % ITSU_LAYERS;
    a.trk_lookup[i] = (layer >= 1 && layer <= ITSU_CELL_LAYERS && count > 0)
                          ? first - a.trk_seg[e * ITSU_TRACKLET_LAYERS + layer]
                          : ITSU_UNUSED_INDEX;
    sid = e * ITSU_TRACKLET_LAYERS + layer;
    if (count > kTrackletSlots) {
      count = 0;
    }
  }
  int total = 0;
  const int excl = warp_exclusive_sum(count, total);
  if (count > 0) {
    w.c[lane] = a.xyzr[i];
    w.owner[lane] = make_int4(first - excl, excl, (int32_t)(i - a.layer_off[seg]), a.layer_off[seg + 1]);
    w.sid[lane] = sid;
  }
  __syncwarp();
  const int32_t *slots = a.trk_slots + (i - lane);
  for (int p0 = 0; p0 < total; p0 += 32) {
    const int p = p0 + lane;
    const int owner = owner_of(excl, p);
    if (p < total) {
      const int4 o = w.owner[owner];
      const int32_t j = slots[(int64_t)(p - o.y) * a.slot_stride + owner];
      const float4 d = a.xyzr[o.w + j];
      const int32_t out = o.x + p;
      if (out % 32 == 0) {
        a.trk_seg32[out / 32] = w.sid[owner];
      }
      store_tracklet(a, out, make_tracklet(w.c[owner], d, o.z, j));
    }
  }
}

// The inner clusters with more than kTrackletSlots tracklets (listed by the count pass, a handful per
// batch) walk their candidates again and write their tracklets in order.
template <bool kGate>
__device__ __forceinline__ void write_crowded(const Arena &a)
{
  const int64_t listed = min(a.status->trk_crowded, (int64_t)a.n_clusters);
  for (int64_t q = global_thread(); q < listed; q += grid_threads()) {
    const int64_t i = a.clu_crowded[q];
    const InnerCluster s = inner_cluster<kGate>(a, i);
    int out = a.trk_off[i];
    walk_inner<kGate>(a, s, [&](int j) { write_tracklet(a, out++, i, s.next_begin + j, s.seg); });
  }
}

// Write pass, part 2, of the stage call (a whole run's segment pass writes them).
template <bool kGate>
__global__ void __launch_bounds__(kMaxThreads) k_tracklets_crowded(Arena a)
{
  if (capacity_failed(a.status)) {
    return;
  }
  write_crowded<kGate>(a);
}

// Cell layer L of event e runs only if tracklet layers 0..L+1 are all non-empty
// (Tracker.cxx:124-128); ts holds the event's first tracklet of each layer and the next event's.
__device__ __forceinline__ bool cells_active(const int32_t *ts, int layer)
{
  for (int l = 0; l <= layer; ++l) {
    if (ts[l + 1] - ts[l] <= 0 || ts[l + 2] - ts[l + 1] <= 0) {
      return false;
    }
  }
  return true;
}

// trk_seg[6e+L] = first tracklet of (e, L); capacity check of the tracklet total. For the cell
// layers, the segment's cell-stage record too (cell_seginfo[2s], [2s+1]): the first cluster of
// layers L, L+1, L+2 (the first -1 when cell layer L of the event does not run), the first
// tracklet of layers L and L+1 and the vertex, so that each first tracklet's setup in the cell
// count pass is two 16-byte loads of one record instead of a dozen loads of per-event offsets.
// crowded: the crowded inner clusters' tracklets too (not in a stage call, whose outputs may still
// have to grow).
template <bool kGate>
__global__ void __launch_bounds__(kCountThreads) k_tracklet_segments(Arena a, bool crowded)
{
  // the cells scan's tile sums start at zero: the cell count pass adds each warp's cells there
  const int64_t n_trk = a.status->total[kTracklets];
  if (n_trk <= a.cap_tracklets) {
    for (int64_t t = global_thread(); t < (n_trk + kScanTile - 1) / kScanTile; t += grid_threads()) {
      a.scan_partials[t] = 0;
    }
  }
  // and so do the segments' cell counts
  for (int64_t s = global_thread(); s < (int64_t)a.n_events * ITSU_CELL_LAYERS; s += grid_threads()) {
    a.cell_seg_count[s] = 0;
  }
  const int nseg = a.n_events * ITSU_TRACKLET_LAYERS;
  for (int s = (int)global_thread(); s <= nseg; s += grid_threads()) {
    if (s == nseg) {
      const int64_t total = a.status->total[kTracklets];
      a.trk_seg[s] = (int32_t)total;
      if (total > a.cap_tracklets) {
        atomicOr(&a.status->flags, kFlagCapTracklets);
      }
    } else {
      const int e = s / ITSU_TRACKLET_LAYERS, layer = s % ITSU_TRACKLET_LAYERS;
      a.trk_seg[s] = a.trk_off[a.layer_off[e * ITSU_LAYERS + layer]];
      if (layer < ITSU_CELL_LAYERS) {
        const int32_t *lo = a.layer_off + e * ITSU_LAYERS;
        int32_t ts[ITSU_LAYERS];
        for (int l = 0; l < ITSU_LAYERS; ++l) {
          ts[l] = a.trk_off[lo[l]];
        }
        const bool active = cells_active(ts, layer);
        a.cell_seginfo[2 * s] = make_int4(active ? lo[layer] : -1, lo[layer + 1], lo[layer + 2], ts[layer]);
        a.cell_seginfo[2 * s + 1] = make_int4(ts[layer + 1], __float_as_int(a.vtx[3 * e]), __float_as_int(a.vtx[3 * e + 1]),
                                              __float_as_int(a.vtx[3 * e + 2]));
      }
    }
  }
  if (crowded && n_trk <= a.cap_tracklets && (*(volatile const int32_t *)&a.status->flags & kFlagCountOverflow) == 0) {
    write_crowded<kGate>(a);
  }
}

// ------------------------------------------------------------------------------------------
// (c) cells: TrackerTraits<false>::computeLayerCells (Tracker.cxx:120-235)

// Count pass. A warp takes a span of 32, 64 or 128 consecutive first tracklets:
//  1. Precut, a lane per first tracklet, 32 at a time: one window per lane (cell_window) against the
//     outgoing tracklets' 4-byte keys, four keys per 16-byte load, about three instructions a pair.
//     The window is a superset of the exact cheap cuts by the keys' resolution; what it lets through
//     (about one pair in eighteen) goes to the warp's queue, in the reference's order (first
//     tracklet, then outgoing tracklet).
//  2. Geometry, a lane per queued pair, in rounds of 32 in the queue's order (a round per group of 32
//     first tracklets would hold 17 pairs on average): the exact cheap cuts (Tracker.cxx:161-173) on
//     the records, then the circle geometry. The passing pairs become the span's cell entries, in
//     order, from the place reserved for the span on (room for all its pairs). Where the scratch is
//     short of that, and has a part for it (cap_cell_pairs), the rounds run twice: the first time they
//     count the cells, which then get exactly their places.
// The cells are counted per span (whose scan places them) and per segment (cell_seg): there is no
// mask, count or offset per tracklet, and the write pass copies entries in order.
// Bound by the gathers (half of the issue slots and of the L1 data pipe busy). Spans of 128 leave
// half a round in five empty, but only pay where every warp has many of them. The grid is one wave of
// resident blocks (9 of 128 threads at 56 registers per SM: a second, part-empty wave would cost
// almost as much again). 1.03 ms per 128 central events; before the prefetch 1.13 (1.15 at 10 blocks
// and 48 registers, 1.21 at 8); as two kernels with the pairs listed in global memory 0.75 + 0.75 ms;
// with masks, counts and lookup entries per first tracklet 1.34 ms, and 0.34 instead of 0.17 ms to
// place the cells.
constexpr int kCellThreads = 128;
constexpr int kCellBlocks = 9;  // resident blocks per SM
constexpr int kMaxSpan = 128;
constexpr int kCellQueue = 512;  // queued pairs of a warp (a span of 128 has 68 on average, 250 behind the tracklet gate)
constexpr int kCellRing = 64;
static_assert(kMaxSpan <= 128 && kMaxMaskedOut <= 64, "a queue item is 7 bits of span and 6 of outgoing tracklets");

// First tracklets in a span, of a run of n. A full grid has 5328 warps (9 blocks of 4 on 148 SMs): from
// 2^20 tracklets on each of them has three spans of 64 or more, from 2^22 six of 128; shorter runs take
// the shortest spans, for as many warps as there are.
__device__ __forceinline__ uint32_t span_of(uint32_t n) { return n >= (1u << 22) ? 128 : (n >= (1u << 20) ? 64 : 32); }

struct CellWarp {
  int2 state[kMaxSpan];        // first outgoing tracklet; segment (kCrowded: more than kMaxMaskedOut outgoing tracklets)
  unsigned long long many;
  union {
    uint16_t queue[kCellQueue];  // (first tracklet in the span) | (outgoing tracklet) << 7
    struct {                     // of a span whose pairs the queue cannot hold
      uint2 ring[kCellRing];     // the same two, for any number of outgoing tracklets
      KeyWindow window[32];      // of 32 first tracklets, and their outgoing ones
      int n_out[32];
    };
  };
};
constexpr int kCrowded = 1 << 30;

// A first tracklet's segment, precut window and outgoing tracklets [j0, j0 + n_out) (none: no cell
// starts with it).
struct CellLane {
  CellWindow w;
  int sid, j0, n_out;
};

__device__ __forceinline__ CellLane cell_lane(const Arena &a, uint32_t k)
{
  CellLane s;
  s.j0 = s.n_out = 0;
  // both loads first: neither depends on the other
  s.sid = tracklet_segment(a, k);
  const itsu_tracklet t1 = load_tracklet(a, k);
  const int layer = s.sid % ITSU_TRACKLET_LAYERS;
  if (layer >= ITSU_CELL_LAYERS) {
    return s;
  }
  const int4 A = a.cell_seginfo[2 * s.sid];
  if (A.x < 0) {
    return s;  // the cell layer does not run
  }
  const int2 out = a.trk_range[A.y + t1.second_cluster];  // the outer cluster's first outgoing tracklet and their number
  const float2 c1 = reinterpret_cast<const float2 *>(a.xyzr + A.x + t1.first_cluster)[1];  // z, r
  s.w = cell_window(t1.tan_lambda, t1.phi, c1.x, c1.y, __int_as_float(a.cell_seginfo[2 * s.sid + 1].w), kC.cell_max_dz[layer]);
  s.j0 = out.x;
  s.n_out = s.w.empty ? 0 : out.y;
  return s;
}

// Which of a lane's outgoing tracklets (1 to kMaxMaskedOut) pass its window. Keys in aligned groups of
// four (the array has room for the last group's overrun): those before j0 fall off by the shift,
// those past the end by the last mask.
__device__ __forceinline__ unsigned long long cell_precut_mask(const Arena &a, const CellLane &s)
{
  const int skip = s.j0 & 3;
  const uint4 *keys = reinterpret_cast<const uint4 *>(a.trk_key + (s.j0 - skip));
  unsigned long long mask = key_window_four(s.w.keys, keys[0]) >> skip;
#pragma unroll 2
  for (int at = 4 - skip; at < s.n_out; at += 4) {
    mask |= (unsigned long long)key_window_four(s.w.keys, *++keys) << at;
  }
  return mask & (~0ull >> (kMaxMaskedOut - s.n_out));
}

// Runs over the spans that end among the tracklets of events below e1 and not below e0 (last: to the
// end of the run): every span is taken once its tracklets are written.
// kExact: the scratch has a part for cells that are counted first (cap_cell_pairs); without one the rounds
// only run once (1.03 ms per 128 central events, 1.06 with the check for it in every span).
template <bool kExact>
__global__ void __launch_bounds__(kCellThreads, kCellBlocks) k_cells_count(Arena a, int32_t e0, int32_t e1, bool last)
{
  __shared__ CellWarp shared[kCellThreads / 32];
  // not stopped by its own scratch flag: the reservations add up to what the run needs
  if ((*(volatile const int32_t *)&a.status->flags & kCapacityMask & ~kFlagCapScratch) != 0) {
    return;
  }
  const int lane = threadIdx.x & 31;
  CellWarp &w = shared[threadIdx.x >> 5];
  w.many = 0;
  // tracklet indices stay below 2^31 (the scan flags larger totals), a span's end below 2^32
  const uint32_t n = (uint32_t)a.status->total[kTracklets];
  const uint32_t span = span_of(n), spans = (n + span - 1) / span;
  const uint32_t s0 = (uint32_t)a.trk_seg[(int64_t)e0 * ITSU_TRACKLET_LAYERS] / span;
  const uint32_t s1 = last ? spans : (uint32_t)a.trk_seg[(int64_t)e1 * ITSU_TRACKLET_LAYERS] / span;
  if (global_thread() == 0) {
    a.status->cell_spans = spans;
  }
  // a whole run's warps take their next spans from a counter (the spans' work differs widely where
  // most pairs pass, as behind the tracklet gate), asked for while the current one is worked on
  const uint32_t warps = gridDim.x * (kCellThreads / 32);
  const bool counter = s0 == 0 && last;
  uint32_t s_next = 0;
  for (uint32_t s = s0 + blockIdx.x * (kCellThreads / 32) + (threadIdx.x >> 5); s < s1; s = s_next) {
    s_next = s + warps;
    if (counter) {
      if (lane == 0) {
        s_next = warps + (uint32_t)atomicAdd(reinterpret_cast<unsigned long long *>(&a.status->cell_next), 1ull);
      }
      s_next = __shfl_sync(0xffffffffu, s_next, 0);
    }
    // The next span's records and keys on their way into L2, a 128-byte line per lane.
    // That span is a round of all warps ahead (two central events), so its data, as first and as
    // outgoing tracklets, is there when its event's spans are worked on (1.125 ms without).
    {
      const int64_t next = (int64_t)s_next * span;
      const void *line = lane < 16 ? (const void *)(a.tracklets + next + lane * 8) : (const void *)(a.trk_key + next + (lane - 16) * 32);
      const uint32_t at = lane < 16 ? lane * 8 : (lane - 16) * 32;
      if (lane < 20 && at < span && next + at < n) {
        prefetch_line(line);
      }
    }
    const uint32_t base = s * span;
    int total = 0;
    bool queued = true;           // the span's pairs are all in the queue
    for (uint32_t g = 0; g < span; g += 32) {
      const uint32_t at = g + lane, k = base + at;
      CellLane p;
      p.sid = p.j0 = p.n_out = 0;
      if (k < n) {
        a.cell_lookup[k] = ITSU_UNUSED_INDEX;  // the write pass fills it for tracklets with cells
        p = cell_lane(a, k);
      }
      const bool crowded = p.n_out > kMaxMaskedOut;
      w.state[at] = make_int2(p.j0, crowded ? p.sid | kCrowded : p.sid);
      unsigned long long mask = 0ull;
      int count = 0;
      if (!crowded && p.n_out > 0) {
        mask = cell_precut_mask(a, p);
        count = __popcll(mask);
      }
      int group_total;
      int to = total + warp_exclusive_sum(count, group_total);
      total += group_total;
      queued = queued && total <= kCellQueue;
      if (__any_sync(0xffffffffu, crowded)) {
        unsigned behind = 0;
        for (int q = 0; crowded && q < p.n_out; ++q) {
          behind += key_window_pass(p.w.keys, a.trk_key[p.j0 + q]);
        }
        const unsigned long long sum = warp_sum(0xffffffffu, behind);
        if (lane == 0) {
          w.many += sum;
        }
        queued = false;
      }
      if (queued) {
        for (unsigned m = (unsigned)mask; m != 0; m &= m - 1u) {
          w.queue[to++] = (uint16_t)(at | (uint32_t)(__ffs(m) - 1) << 7);
        }
        for (unsigned m = (unsigned)(mask >> 32); m != 0; m &= m - 1u) {
          w.queue[to++] = (uint16_t)(at | (uint32_t)(__ffs(m) + 31) << 7);
        }
      }
    }
    unsigned cells = 0;
    unsigned long long first = 0;
    __syncwarp();
    const unsigned long long pairs = queued ? (unsigned long long)total : w.many + (unsigned)total;
    bool placed = false, counting = false;
    if (pairs > 0) {
      if (lane == 0) {
        first = atomicAdd(reinterpret_cast<unsigned long long *>(&a.status->cell_entries), pairs);
      }
      first = __shfl_sync(0xffffffffu, first, 0);
      placed = first + pairs <= (unsigned long long)a.cap_cell_pairs;
      counting = kExact && !placed;
      if (lane == 0 && !placed && !counting) {
        atomicOr(&a.status->flags, kFlagCapScratch);  // nothing after this pass runs
      }
    }
    while (placed || (kExact && counting)) {
      __syncwarp();
      unsigned head = 0, tail = queued ? total : 0;
      // not queued (a crowded outer cluster, or more pairs than the queue holds): the first tracklets' keys are
      // walked again, 32 of one tracklet at a time, against windows made 32 at a time (64 events of 300
      // clusters per layer on a line, 11.6 million tracklets: 12.9 ms; 18.8 with each window made by the warp)
      uint32_t next = queued ? span : 0, next_out = 0;
      for (;;) {
        if (next < span && tail - head < 32) {
          const uint32_t of = next & 31u;
          if (of == 0 && next_out == 0) {  // the next 32 first tracklets' windows, a lane each
            const uint32_t k = base + next + lane;
            CellLane p;
            p.j0 = p.n_out = 0;
            if (k < n) {
              p = cell_lane(a, k);
            }
            w.window[lane] = p.w.keys;
            w.n_out[lane] = p.n_out;
            __syncwarp();
          }
          const uint32_t q = next_out + lane, n_out = (uint32_t)w.n_out[of];
          const bool listed = q < n_out && key_window_pass(w.window[of], a.trk_key[(uint32_t)w.state[next].x + q]);
          const unsigned m = __ballot_sync(0xffffffffu, listed);
          if (listed) {
            w.ring[(tail + __popc(m & ((1u << lane) - 1u))) & (kCellRing - 1)] = make_uint2(next, q);
          }
          tail += __popc(m);
          next_out += 32;
          if (next_out >= n_out) {
            next_out = 0;
            ++next;
          }
          __syncwarp();
          continue;
        }
        const unsigned m = min(tail - head, 32u);
        if (m == 0) {
          break;
        }
        bool pass = false, crowded = false;
        int sid = 0, segment = 0;
        uint32_t k = 0, j = 0;
        itsu_tracklet f, t;
        int4 A, B;
        float3 normal;
        float curvature, dca;
        if (lane < (int)m) {
          uint2 item;  // place of the first tracklet in the span, and which outgoing tracklet
          if (queued) {
            const uint32_t packed = w.queue[head + lane];
            item = make_uint2(packed & 127u, packed >> 7);
          } else {
            item = w.ring[(head + lane) & (kCellRing - 1)];
          }
          const uint32_t at = item.x;
          const int2 state = w.state[at];
          crowded = (state.y & kCrowded) != 0;
          sid = state.y & ~kCrowded;
          k = base + at;
          j = (uint32_t)state.x + item.y;
          A = a.cell_seginfo[2 * sid];
          B = a.cell_seginfo[2 * sid + 1];
          f = load_tracklet(a, k);
          t = load_tracklet(a, j);
          const float4 c1 = a.xyzr[A.x + f.first_cluster];
          const float4 c2 = a.xyzr[A.y + f.second_cluster];
          const float4 c3 = a.xyzr[A.z + t.second_cluster];
          const int e = sid / ITSU_TRACKLET_LAYERS, layer = sid - e * ITSU_TRACKLET_LAYERS;
          segment = sid - e;  // 5 e + layer
          pass = cell_precut(layer, f.tan_lambda, f.phi, t.tan_lambda, t.phi, c1, __int_as_float(B.w)) &&
                 cell_geometry(layer, c1, c2, c3, __int_as_float(B.y), __int_as_float(B.z), normal, curvature, dca);
        }
        head += m;
        const unsigned passed = __ballot_sync(0xffffffffu, pass);
        const unsigned same = __match_any_sync(0xffffffffu, pass ? segment : -1);
        if (pass && !(kExact && counting)) {
          const unsigned before = (1u << lane) - 1u;
          if ((same & before) == 0) {
            atomicAdd(&a.cell_seg_count[segment], __popc(same));
          }
          const int64_t slot = (int64_t)first + cells + __popc(passed & before);
          int2 *dst = reinterpret_cast<int2 *>(a.cell_entries + slot);
          dst[0] = make_int2(f.first_cluster, f.second_cluster);
          dst[1] = make_int2(t.second_cluster, (int)(k - (uint32_t)A.w));
          dst[2] = make_int2((int)(j - (uint32_t)B.x), __float_as_int(normal.x));
          dst[3] = make_int2(__float_as_int(normal.y), __float_as_int(normal.z));
          dst[4] = make_int2(__float_as_int(curvature), crowded ? segment | kEntryUnscored : segment);
          if (a.mlp) {
            a.cell_dca[slot] = dca;
          }
        }
        cells += __popc(passed);
        __syncwarp();  // the queue's freed places are refilled
      }
      if (!kExact || !counting) {
        break;
      }
      counting = false;
      if (cells > 0) {
        if (lane == 0) {
          first = a.cap_cell_pairs + atomicAdd(reinterpret_cast<unsigned long long *>(&a.status->cell_exact), (unsigned long long)cells);
        }
        first = __shfl_sync(0xffffffffu, first, 0);
        placed = first + cells <= (unsigned long long)a.cap_cell_entries;
        if (lane == 0 && !placed) {
          atomicOr(&a.status->flags, kFlagCapScratch);
        }
        cells = 0;
      }
    }
    if (lane == 0) {
      a.cell_span[s] = make_uint2((unsigned)first, cells);  // within cap_cell_entries (kMaxCellEntries at most)
      a.cell_span_count[s] = (int32_t)cells;
      if (cells > INT_MAX) {
        atomicOr(&a.status->flags, kFlagCountOverflow);
      }
      if (cells > 0) {
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.scan_partials[s / kScanTile]), (unsigned long long)cells);
      }
    }
    if (lane == 0 && !queued) {
      w.many = 0;
    }
    __syncwarp();  // the span's state is refilled next
  }
}

// The place of the p-th entry of a warp's spans (each lane has one: its first entry and the prefix sum of
// the lanes' entries before it), and the lane whose span it is of. All lanes call it together. Entries are
// counted in 32 unsigned bits: the scratch holds kMaxCellEntries of them at most.
__device__ __forceinline__ int64_t span_entry(unsigned first, unsigned excl, unsigned p, int &owner)
{
  owner = owner_of(excl, p);
  return (int64_t)__shfl_sync(0xffffffffu, first, owner) + p - __shfl_sync(0xffffffffu, excl, owner);
}

// Learned prefilter: scores the cell entries, 32 per warp on the tensor cores, and drops those whose
// logit is below the model's threshold (entry and counts) before the scan. The score and the exact
// cuts are combined with AND, so scoring only the pairs that passed the cuts (whose geometry also
// gave the DCA feature) keeps the same cells as scoring every candidate first. A NaN logit keeps its
// cell. The pairs of a tracklet with more than kMaxMaskedOut outgoing tracklets are kept unscored.
// A warp takes consecutive spans and flattens their entries over its lanes, so that the network's
// tiles are full: about three times in all, the same number for every warp (one wave of blocks, 24
// warps per SM). Bound by the network's activations: 0.154 ms per 32 central events; 0.175 in blocks
// of 256 threads with 2^13 turns shared out unevenly.
constexpr int kPrefilterThreads = 128;
constexpr int kPrefilterBlocks = 6;  // resident blocks per SM, by registers
constexpr int kPrefilterTurns = 3;

__global__ void __launch_bounds__(kPrefilterThreads, kPrefilterBlocks) k_cells_prefilter(Arena a)
{
  __shared__ MlpSmem mlp;
  __shared__ __align__(16) __nv_bfloat16 rows[kPrefilterThreads / 32][32][kRowPitch];
  load_mlp(mlp, *a.mlp);
  __syncthreads();
  if (capacity_failed(a.status)) {
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t spans = a.status->cell_spans;
  const int64_t turns = (int64_t)gridDim.x * (kPrefilterThreads / 32) * kPrefilterTurns;
  const int take = (int)min((int64_t)32, (spans + turns - 1) / turns);  // spans at a time
  for (int64_t s0 = ((int64_t)blockIdx.x * (kPrefilterThreads / 32) + warp) * take; s0 < spans;
       s0 += (int64_t)gridDim.x * (kPrefilterThreads / 32) * take) {
    const uint2 in = lane < take && s0 + lane < spans ? a.cell_span[s0 + lane] : make_uint2(0, 0);  // first entry, entries
    unsigned total;
    const unsigned excl = warp_exclusive_sum(in.y, total);
    for (unsigned p0 = 0; p0 < total; p0 += 32) {
      const unsigned p = p0 + lane;
      int owner;
      const int64_t i = span_entry(in.x, excl, p, owner);
      int segment = kEntryUnscored;
      int2 h0, h1, h2;
      if (p < total) {
        const int2 *src = reinterpret_cast<const int2 *>(a.cell_entries + i);
        h0 = src[0], h1 = src[1], h2 = src[2], segment = src[4].y;
      }
      float f[kMlpIn];
      const bool scored = !(segment & kEntryUnscored);
      if (scored) {
        const int layer = segment % ITSU_CELL_LAYERS, sid = segment + segment / ITSU_CELL_LAYERS;  // 6 e + layer
        const int4 A = a.cell_seginfo[2 * sid], B = a.cell_seginfo[2 * sid + 1];
        const itsu_tracklet t1 = load_tracklet(a, A.w + h1.y);
        const itsu_tracklet t2 = load_tracklet(a, B.x + h2.x);
        const float4 c1 = a.xyzr[A.x + h0.x];
        const float4 c2 = a.xyzr[A.y + h0.y];
        const float4 c3 = a.xyzr[A.z + h1.x];
        pair_features(layer, t1.tan_lambda, t1.phi, t2.tan_lambda, t2.phi, c1, c2, c3, __int_as_float(B.y), __int_as_float(B.z),
                      __int_as_float(B.w), a.cell_dca[i], f);
      } else {
        for (int k = 0; k < kMlpIn; ++k) {
          f[k] = mlp.mean[k];
        }
      }
      feature_row(mlp.mean, mlp.inv_std, f, rows[warp][lane]);
      __syncwarp();
      const float logit = mlp_logits_warp(mlp, rows[warp]);
      if (scored && logit < mlp.threshold) {
        a.cell_entries[i].segment = kEntryDropped;
        atomicSub(&a.cell_span_count[s0 + owner], 1);
        atomicSub(&a.cell_seg_count[segment], 1);
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.scan_partials[(s0 + owner) / kScanTile]), ~0ull);  // its tile sum - 1
      }
      __syncwarp();
    }
  }
}

// Write pass: a warp takes consecutive spans (a span of 128 has 15 entries in central events, 85 behind
// the tracklet gate) and flattens their entries over its lanes; in order, they go to the spans' scanned
// places, which are contiguous (a dropped entry leaves no gap). The first cell of each first tracklet
// fills its cells lookup entry, and each cell's state of the stages after is reset (the neighbour
// scan's tile sums too). Many turns keep many stores in flight (0.18 ms per 128 central events; with
// 2^13 turns 0.20; with the next turn's entries prefetched 0.20).
constexpr int kScatterThreads = 256;
constexpr int64_t kScatterTurns = 1 << 16;

// A cell's CA level and its number of level-decreasing chains down to layer 0, in one word
// (chains << 3 | level; levels are 1..5 and chain counts are capped at INT_MAX), of layers 1 to 4; the
// cells of layer 0 all have level 1 and one chain.
__device__ __forceinline__ int64_t chain_word(int64_t paths, int level) { return (paths << 3) | level; }
__device__ __forceinline__ int chain_level(int64_t w) { return (int)(w & 7); }
__device__ __forceinline__ int64_t chain_paths(int64_t w) { return w >> 3; }

// A cell's state of the neighbour and road stages before they run.
__device__ __forceinline__ void reset_cell(const Arena &a, int64_t c)
{
  a.nb_count[c] = 0;
  a.road_count[c] = 0;
}

__device__ __forceinline__ void zero_tiles(int64_t *partials, int64_t n)
{
  for (int64_t t = global_thread(); t < (n + kScanTile - 1) / kScanTile; t += grid_threads()) {
    partials[t] = 0;
  }
}

__global__ void __launch_bounds__(kScatterThreads) k_cells_scatter(Arena a)
{
  if (capacity_failed(a.status)) {
    return;
  }
  zero_tiles(a.scan_partials, a.status->total[kCells]);
  const int lane = threadIdx.x & 31;
  const int64_t spans = a.status->cell_spans;
  const int take = (int)min((int64_t)32, max((int64_t)1, spans / kScatterTurns));  // spans at a time
  for (int64_t s0 = ((int64_t)blockIdx.x * (kScatterThreads / 32) + (threadIdx.x >> 5)) * take; s0 < spans;
       s0 += (int64_t)gridDim.x * (kScatterThreads / 32) * take) {
    const uint2 in = lane < take && s0 + lane < spans ? a.cell_span[s0 + lane] : make_uint2(0, 0);  // first entry, entries
    unsigned total;
    const unsigned excl = warp_exclusive_sum(in.y, total);
    int out0 = a.cell_span_off[s0];
    int last_t1 = -1, last_segment = -1;  // of the cell before
    for (unsigned p0 = 0; p0 < total; p0 += 32) {
      const unsigned p = p0 + lane;
      int owner;
      const int64_t i = span_entry(in.x, excl, p, owner);
      int2 h[5];
      h[1].y = 0;
      h[4].y = kEntryDropped;
      if (p < total) {
        const int2 *src = reinterpret_cast<const int2 *>(a.cell_entries + i);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          h[q] = src[q];
        }
      }
      const bool alive = h[4].y != kEntryDropped;
      const unsigned living = __ballot_sync(0xffffffffu, alive);
      if (living == 0) {
        continue;
      }
      const unsigned before = living & ((1u << lane) - 1u);
      const int out = out0 + __popc(before);
      const int segment = h[4].y & ~kEntryUnscored, t1 = h[1].y;
      const int from = before ? 31 - __clz(before) : 0;
      const int t1_before = __shfl_sync(0xffffffffu, t1, from), segment_before = __shfl_sync(0xffffffffu, segment, from);
      if (alive) {
        const bool first = before ? (t1_before != t1 || segment_before != segment) : (last_t1 != t1 || last_segment != segment);
        const int e = segment / ITSU_CELL_LAYERS, layer = segment % ITSU_CELL_LAYERS;
        if (first && layer >= 1) {
          a.cell_lookup[a.trk_seg[e * ITSU_TRACKLET_LAYERS + layer] + t1] = out - a.cell_seg[segment];
        }
        int2 *dst = reinterpret_cast<int2 *>(a.cells + out);
        h[4].y = 1;  // level
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          dst[q] = h[q];
        }
        a.cell_seg_id[out] = segment;
        reset_cell(a, out);
      }
      const int to = 31 - __clz(living);
      last_t1 = __shfl_sync(0xffffffffu, t1, to);
      last_segment = __shfl_sync(0xffffffffu, segment, to);
      out0 += __popc(living);
    }
  }
}

// cell_seg[5e+L] = first cell of (e, L), from the segments' counts (cells are in segment order), by
// one block.
__device__ void cell_segments(const Arena &a, int64_t *warp_totals)
{
  constexpr int kPer = 4;
  const int nseg = a.n_events * ITSU_CELL_LAYERS;
  int64_t carry = 0;
  for (int s0 = 0; s0 < nseg; s0 += kPer * (int)blockDim.x) {
    const int s = s0 + kPer * (int)threadIdx.x;
    int32_t v[kPer];
    int64_t sum = 0, total;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      v[k] = s + k < nseg ? a.cell_seg_count[s + k] : 0;
      sum += v[k];
    }
    int64_t run = carry + block_exclusive_scan<int64_t>(sum, warp_totals, total);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      if (s + k < nseg) {
        a.cell_seg[s + k] = (int32_t)run;
      }
      run += v[k];
    }
    carry += total;
  }
  if (threadIdx.x == 0) {
    a.cell_seg[nseg] = (int32_t)carry;
  }
}

// ------------------------------------------------------------------------------------------
// (d) neighbours and CA levels: Tracker<IsGPU>::findCellsNeighbours (Tracker.cxx:417-474)

// Stage call only: the cells' state again, so that the stage can be re-run.
__global__ void __launch_bounds__(kMaxThreads) k_neighbour_reset(Arena a)
{
  if (capacity_failed(a.status)) {
    return;
  }
  const int64_t n = a.status->total[kCells];
  for (int64_t c = global_thread(); c < n; c += grid_threads()) {
    reset_cell(a, c);
  }
}

// Tracker.cxx:416-474 (findCellsNeighbours): a cell of layer L and the cells of layer L + 1 built
// on its second tracklet (from its cells lookup entry on, as long as they are built on it). The
// count pass evaluates the cut, counts each passing pair in its row and keeps the first candidate and
// the passing ones as a mask (of up to kMaskedRun candidates; a longer run is marked in the top bit);
// the write pass, after the scan of the counts, fills the rows from these (re-evaluating the cut only
// for the marked cells), counting the counts down to zero. Row order is restored by k_levels' sort.
// Bound by the latency of the gathers: 0.118 and 0.065 ms per 128 central events; the write pass took
// 0.095 when it looked the first candidate up again through the cell's record.
constexpr int kMaskedRun = 63;
constexpr unsigned long long kLongRun = 1ull << kMaskedRun;

template <bool kWrite>
__global__ void __launch_bounds__(kMaxThreads) k_neighbours(Arena a)
{
  if (capacity_failed(a.status)) {
    return;
  }
  const int64_t n = a.status->total[kCells];
  if (kWrite) {
    zero_tiles(a.road_partials, n);  // the level pass adds each tile's roads
  }
  for (int64_t c = global_thread(); c < n; c += grid_threads()) {
    const int sid = a.cell_seg_id[c];
    const int e = sid / ITSU_CELL_LAYERS, layer = sid % ITSU_CELL_LAYERS;
    if (layer >= ITSU_NEIGHBOUR_LAYERS) {
      continue;
    }
    const int32_t c_local = (int32_t)(c - a.cell_seg[sid]);
    if (kWrite) {
      unsigned long long mask = a.nb_mask[c];
      const int32_t j0 = a.nb_first[c];
      if (!(mask & kLongRun)) {
        for (; mask; mask &= mask - 1ull) {
          const int32_t j = j0 + __ffsll((long long)mask) - 1;
          const int slot = atomicSub(&a.nb_count[j], 1) - 1;
          a.nb[a.nb_off[j] + slot] = c_local;
        }
        continue;
      }
    }
    unsigned long long mask = 0ull;
    const int32_t second = a.cells[c].second_tracklet;
    const int32_t found = a.cell_lookup[a.trk_seg[e * ITSU_TRACKLET_LAYERS + layer + 1] + second];
    const int32_t j0 = a.cell_seg[sid + 1] + found, j1 = found < 0 ? j0 : a.cell_seg[sid + 2];
    const itsu_cell cell = a.cells[c];
    const float3 n1 = make_float3(cell.nx, cell.ny, cell.nz);
    int links = 0;  // to cells of j0's scan tile
    for (int32_t j = j0; j < j1; ++j) {
      const itsu_cell next = a.cells[j];
      if (next.first_tracklet != second) {
        break;
      }
      const bool pass = neighbour_cut(layer, n1, cell.curvature, make_float3(next.nx, next.ny, next.nz), next.curvature);
      if (kWrite) {
        if (pass) {
          const int slot = atomicSub(&a.nb_count[j], 1) - 1;
          a.nb[a.nb_off[j] + slot] = c_local;
        }
      } else {
        if (pass) {
          atomicAdd(&a.nb_count[j], 1);
          if (j / kScanTile == j0 / kScanTile) {
            ++links;
          } else {
            atomicAdd(reinterpret_cast<unsigned long long *>(&a.scan_partials[j / kScanTile]), 1ull);
          }
        }
        if (j - j0 >= kMaskedRun) {
          mask |= kLongRun;
        } else if (pass) {
          mask |= 1ull << (j - j0);
        }
      }
    }
    if (!kWrite) {
      a.nb_mask[c] = mask;
      a.nb_first[c] = j0;
      if (links > 0) {
        add_to_tile(a.scan_partials, j0, links);
      }
    }
  }
}

// One cell of k_levels (below): its row sorted, its level and its number of chains (read from and
// written to the neighbours' chain words, one 8-byte gather per neighbour).
__device__ __forceinline__ void level_of(const Arena &a, int64_t c, int64_t prev_base, int layer)
{
  const int32_t b = a.nb_off[c], en = a.nb_off[c + 1];
  int32_t *row = a.nb + b;
  int len = en - b;
  for (int p = 1; p < len; ++p) {
    const int32_t v = row[p];
    int q = p - 1;
    while (q >= 0 && row[q] > v) {
      row[q + 1] = row[q];
      --q;
    }
    row[q + 1] = v;
  }
  int level = 1;
  int64_t paths = 0;
  bool overflow = false;
  if (layer == 1) {  // every neighbour has level 1 and one chain
    level = len > 0 ? 2 : 1;
    paths = len;
    len = 0;
  }
  for (int p = 0; p < len; ++p) {
    level = max(level, chain_level(a.paths[prev_base + row[p]]) + 1);
  }
  for (int p = 0; p < len; ++p) {
    const int64_t w = a.paths[prev_base + row[p]];
    if (chain_level(w) == level - 1) {
      paths += chain_paths(w);
      if (paths > INT_MAX) {
        paths = INT_MAX;
        overflow = true;
      }
    }
  }
  a.cells[c].level = level;
  a.paths[c] = chain_word(paths, level);
  if (layer == ITSU_CELL_LAYERS - 1 && level == kCellsMinLevel) {
    a.road_count[c] = (int32_t)paths;
    if (paths > 0) {
      add_to_tile(a.road_partials, c, (int)paths);
    }
    if (overflow) {
      atomicOr(&a.status->flags, kFlagCountOverflow);
    }
  }
}

// Layer by layer from 1: rows sorted ascending (the reference pushes in cell order), then the level
// (Tracker.cxx:463-468: 1 + the highest neighbour level) and the number of level-decreasing chains
// down to layer 0 (the roads a level-5 cell starts, Tracker.cxx:477-571). A cluster of CTAs per event
// (events beyond the grid in turn), which meet after each layer: one launch in place of four.
template <int kThreads_>
__global__ void __launch_bounds__(kThreads_) k_levels(Arena a)
{
  namespace cg = cooperative_groups;
  const int ctas = (int)cg::this_cluster().num_blocks(), rank = (int)cg::this_cluster().block_rank();
  if (capacity_failed(a.status)) {
    return;  // a thread that finds a count overflow of this pass here leaves; the barriers wait for the others only
  }
  for (int e = blockIdx.x / ctas; e < a.n_events; e += gridDim.x / ctas) {
    const int32_t *cs = a.cell_seg + e * ITSU_CELL_LAYERS;
    for (int layer = 1; layer < ITSU_CELL_LAYERS; ++layer) {
      const int64_t prev_base = cs[layer - 1];
      for (int64_t c = cs[layer] + rank * kThreads_ + (int)threadIdx.x; c < cs[layer + 1]; c += ctas * kThreads_) {
        level_of(a, c, prev_base, layer);
      }
      if (layer < ITSU_CELL_LAYERS - 1) {
        if (ctas == 1) {
          __syncthreads();
        } else {
          cg::this_cluster().sync();
        }
      }
    }
  }
}

// One layer of the level pass over the whole chip (the blocks of grid row y take events y, y + gridDim.y,
// ...): for few events whose layers are more than a cluster of CTAs takes in a few rounds (level_shape).
__global__ void __launch_bounds__(kMaxThreads) k_levels_layer(Arena a, int layer)
{
  if (capacity_failed(a.status)) {
    return;
  }
  for (int e = blockIdx.y; e < a.n_events; e += gridDim.y) {
    const int32_t *cs = a.cell_seg + e * ITSU_CELL_LAYERS;
    const int64_t prev_base = cs[layer - 1];
    for (int64_t c = cs[layer] + global_thread(); c < cs[layer + 1]; c += grid_threads()) {
      level_of(a, c, prev_base, layer);
    }
  }
}

// ------------------------------------------------------------------------------------------
// (e) roads: Tracker<IsGPU>::findTracks / traverseCellsTree / computeMontecarloLabels

// A sorted cluster's MC id, from its 16-byte auxiliary record (the batch's 36-byte sorted records
// are twice the footprint, and the road vote's gathers hit L2 less often there).
__device__ __forceinline__ int32_t cluster_mc(const Arena &a, const int32_t *lo, int layer, int32_t idx)
{
  return a.clu_aux[lo[layer] + idx].z;
}

// One road per lane: the roads of a warp's 32 consecutive cells form one contiguous range (the
// scan of the roots' chain counts), which the lanes fill together, each lane taking the next road
// of the range, finding its root cell (owner) and its rank k among the root's roads. The traversal
// of Tracker.cxx:477-571 visits a cell's neighbours in row order and descends into those one level
// down, so the root's k-th road is found by walking down the layers: at each, skip the neighbours
// one level down whose whole subtrees (their chain counts, k_levels) lie before k, and descend into
// the one holding it. A complete chain is labelled by Moore's vote over its 7 clusters
// (Tracker.cxx:574-652) and stored with coalesced writes. The roots are the last layer's cells:
// the blocks of grid row y take those of events y, y + gridDim.y, ...
__global__ void __launch_bounds__(kMaxThreads) k_roads(Arena a)
{
  if (capacity_failed(a.status)) {
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (int e = blockIdx.y; e < a.n_events; e += gridDim.y) {
    const int32_t *cs = a.cell_seg + e * ITSU_CELL_LAYERS;
    const int32_t *lo = a.layer_off + e * ITSU_LAYERS;
    const int64_t n = cs[ITSU_CELL_LAYERS];  // the event's last cell + 1
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // the event's first road
      a.road_seg[e] = a.road_off[cs[ITSU_CELL_LAYERS - 1]];
      if (e == a.n_events - 1) {
        a.road_seg[e + 1] = (int32_t)a.status->total[kRoads];
      }
    }
    for (int64_t base = cs[ITSU_CELL_LAYERS - 1] + warp * 32; base < n; base += warps * 32) {
      const int64_t c = base + lane;
      int32_t first = 0, count = 0;
      if (c < n) {
        first = a.road_off[c];
        count = a.road_off[c + 1] - first;
      }
      int total = 0;
      const int excl = warp_exclusive_sum(count, total);
      if (total == 0) {
        continue;
      }
      const int64_t out0 = __shfl_sync(0xffffffffu, first, 0);
      for (int p0 = 0; p0 < total; p0 += 32) {
        const int p = p0 + lane;
        const int owner = owner_of(excl, p);
        int64_t k = p - __shfl_sync(0xffffffffu, excl, owner);
        if (p >= total) {
          continue;
        }
        int64_t flat = base + owner;
        int32_t cur[ITSU_CELL_LAYERS];  // local cell index per layer along the chain
        cur[ITSU_CELL_LAYERS - 1] = (int32_t)(flat - cs[ITSU_CELL_LAYERS - 1]);
        int level = kCellsMinLevel;
        bool found = true;
#pragma unroll
        for (int l = ITSU_CELL_LAYERS - 1; l >= 2; --l) {
          const int32_t j1 = a.nb_off[flat + 1];
          bool down = false;
          cur[l - 1] = 0;
          for (int32_t j = a.nb_off[flat]; j < j1; ++j) {
            const int32_t nb = a.nb[j];
            const int64_t nflat = cs[l - 1] + nb;
            const int64_t w = a.paths[nflat];
            if (chain_level(w) == level - 1) {
              const int64_t below = chain_paths(w);
              if (k < below) {
                cur[l - 1] = nb;
                flat = nflat;
                down = true;
                break;
              }
              k -= below;
            }
          }
          found = found && down;
          --level;
        }
        {  // layer 1 to 0: every neighbour has one chain
          const int32_t j0 = a.nb_off[flat], j1 = a.nb_off[flat + 1];
          const bool down = found && k < j1 - j0;
          cur[0] = down ? a.nb[j0 + k] : 0;
          found = down;
        }
        if (!found) {  // only when a chain count was capped (the count overflow flag is set)
          atomicOr(&a.status->flags, kFlagCountOverflow);
        }
        itsu_road road;
        int max_value = ITSU_UNUSED_INDEX, votes = 0;
        bool fake = false;
#pragma unroll
        for (int l = 0; l < ITSU_CELL_LAYERS; ++l) {
          road.cell_ids[l] = cur[l];
          const itsu_cell &cell = a.cells[cs[l] + cur[l]];
          if (l == 0) {
            max_value = cluster_mc(a, lo, 0, cell.first_cluster);
            votes = 1;
            const int second = cluster_mc(a, lo, 1, cell.second_cluster);
            if (second == max_value) {
              ++votes;
            } else {
              max_value = second;
              votes = 1;
              fake = true;
            }
          }
          const int current = cluster_mc(a, lo, l + 2, cell.third_cluster);
          if (current == max_value) {
            ++votes;
          } else {
            --votes;
            fake = true;
          }
          if (votes == 0) {
            max_value = current;
            votes = 1;
          }
        }
        road.size = ITSU_CELL_LAYERS;
        road.label = max_value;
        road.is_fake = fake ? 1 : 0;
        road.pad_[0] = road.pad_[1] = road.pad_[2] = 0;
        a.roads[out0 + p] = road;
      }
    }
  }
}

__global__ void k_atan2f(const float *y, const float *x, float *out, int64_t n)
{
  for (int64_t i = global_thread(); i < n; i += grid_threads()) {
    out[i] = itsu_atan2f(y[i], x[i]);
  }
}

// Grid of the grid-stride kernels: the tuned number of resident blocks per SM, scaled to the
// block size so that the number of resident threads stays comparable.
int fixed_grid(const Launch &l) { return l.num_sms * l.blocks_per_sm; }

// Grid of the per-event kernels (a row of blocks per event, events beyond 65535 rows taken in
// turn): about the same blocks in all as the grid-stride kernels.
dim3 event_grid(const Arena &a, const Launch &l)
{
  const int rows = std::min(a.n_events, 65535);
  const int64_t full = std::max(1, (fixed_grid(l) + rows - 1) / rows);
  return dim3(blocks_for(full, l.cells / std::max(rows, 1), l.block), (unsigned)rows);
}

void step_status_init(const Arena &a, const Launch &l)
{
  const int64_t tiles = (a.n_clusters + kScanTile - 1) / kScanTile;
  const int64_t blocks = a.scan_partials ? std::min<int64_t>((tiles + kThreads - 1) / kThreads, l.num_sms) : 0;
  k_status_init<<<(unsigned)std::max<int64_t>(blocks, 1), kThreads, 0, l.stream>>>(a);
}

// A launch of `ctas` CTAs per cluster (1: no cluster).
template <typename... Args>
void launch_clusters(void (*kernel)(Args...), int64_t clusters, int ctas, int threads, size_t bytes, cudaStream_t stream, Args... args)
{
  cudaLaunchConfig_t config{};
  config.gridDim = dim3((unsigned)(clusters * ctas));
  config.blockDim = dim3((unsigned)threads);
  config.dynamicSmemBytes = bytes;
  config.stream = stream;
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = (unsigned)ctas;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  config.attrs = &cluster;
  config.numAttrs = ctas > 1 ? 1 : 0;
  cudaLaunchKernelEx(&config, kernel, args...);
}

template <int kThreads_>
void launch_sort(const Arena &a, const Launch &l, int ctas)
{
  const size_t bytes = sort_shared_bytes(kThreads_ / 32);
  if (bytes > 48 * 1024) {
    cudaFuncSetAttribute(k_cluster_sort<kThreads_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  }
  launch_clusters(k_cluster_sort<kThreads_>, (int64_t)a.n_events * ITSU_LAYERS, ctas, kThreads_, bytes, l.stream, a);
}

void step_cluster_sort(const Arena &a, const Launch &l)
{
  if (a.n_events <= 0) {
    return;
  }
  const SortShape shape = sort_shape(a.n_events, a.n_clusters, l.max_segment);
  if (shape.threads == 64) {
    launch_sort<64>(a, l, shape.ctas);
  } else if (shape.threads == 256) {
    launch_sort<256>(a, l, shape.ctas);
  } else {
    launch_sort<512>(a, l, shape.ctas);
  }
}

// The per-item count passes need whole warps: each warp adds its items' total to one scan tile.
bool whole_warps(const Arena &a, const Launch &l)
{
  if (l.block % 32 == 0) {
    return true;
  }
  k_flag_bad_launch<<<1, 1, 0, l.stream>>>(a.status);
  return false;
}

void step_tracklets_count(const Arena &a, const Launch &l)
{
  if (!whole_warps(a, l)) {
    return;
  }
  const int64_t blocks = (a.n_clusters + l.block - 1) / l.block;
  if (blocks <= 0) {
    return;
  }
  // the count pass takes at most kCountThreads threads per block (any whole warps give the same
  // results)
  const int block = std::min(l.block, kCountThreads);
  const unsigned grid = (unsigned)((a.n_clusters + block - 1) / block);
  if (a.gate) {
    k_tracklets_count<true><<<grid, block, 0, l.stream>>>(a);
  } else {
    k_tracklets_count<false><<<grid, block, 0, l.stream>>>(a);
  }
}

// Launches only in the learned form with the tracklet gate (a.gate set).
void step_tracklets_gate(const Arena &a, const Launch &l)
{
  if (a.gate && a.n_clusters > 0 && a.n_events > 0) {
    const int rows = std::min(a.n_events, 65535);
    const int per_event = std::max(1, (l.num_sms * 8 + rows - 1) / rows);
    k_tracklets_gate<<<dim3((unsigned)per_event, (unsigned)rows), kGateThreads, 0, l.stream>>>(a);
  }
}

void launch_write_range(const Arena &a, const Launch &l, int64_t c0, int64_t c1)
{
  const int64_t blocks = (c1 - c0 + kWriteThreads - 1) / kWriteThreads;
  if (blocks > 0) {
    k_tracklets_write<<<(unsigned)blocks, kWriteThreads, 0, l.stream>>>(a, c0, c1);
  }
}

// The write and cell count passes over all events at once (launches with no event groups).
void step_tracklets_write(const Arena &a, const Launch &l)
{
  if (l.n_groups == 0) {
    launch_write_range(a, l, 0, a.n_clusters);
  }
}

// A whole run's crowded clusters are written by the segment pass.
void step_tracklets_crowded(const Arena &a, const Launch &l)
{
  if (!l.staged) {
    return;
  }
  if (a.gate) {
    k_tracklets_crowded<true><<<l.num_sms, 128, 0, l.stream>>>(a);
  } else {
    k_tracklets_crowded<false><<<l.num_sms, 128, 0, l.stream>>>(a);
  }
}

// Blocks for the segments, and a thread per cluster, any of which may be crowded.
unsigned segment_blocks(const Arena &a, const Launch &l) { return blocks_for(l.num_sms, a.n_events * ITSU_TRACKLET_LAYERS + a.n_clusters, 128); }

void step_tracklet_segments(const Arena &a, const Launch &l)
{
  if (a.gate) {
    k_tracklet_segments<true><<<segment_blocks(a, l), 128, 0, l.stream>>>(a, !l.staged);
  } else {
    k_tracklet_segments<false><<<segment_blocks(a, l), 128, 0, l.stream>>>(a, !l.staged);
  }
}

void launch_cells_range(const Arena &a, const Launch &l, int32_t e0, int32_t e1, bool last)
{
  const unsigned blocks = blocks_for(l.num_sms * kCellBlocks, l.tracklets, kCellThreads);
  if (a.cap_cell_pairs < a.cap_cell_entries) {
    k_cells_count<true><<<blocks, kCellThreads, 0, l.stream>>>(a, e0, e1, last);
  } else {
    k_cells_count<false><<<blocks, kCellThreads, 0, l.stream>>>(a, e0, e1, last);
  }
}

void step_cells_count(const Arena &a, const Launch &l)
{
  if (l.n_groups == 0) {
    launch_cells_range(a, l, 0, a.n_events, true);
  }
}

// Event groups: the write pass of a group's inner clusters, then the cell count pass of its
// tracklets, group after group, so that the tracklets a group's count pass gathers were written
// moments before and are still in L2. Group g's clusters are [groups[g], groups[g + 1]) (multiples
// of 32 up to the last), its events [g * group_events, (g + 1) * group_events). A span that reaches
// into the next group's tracklets is left to that group.
void step_write_count_groups(const Arena &a, const Launch &l)
{
  if (l.n_groups == 0 || !whole_warps(a, l)) {
    return;
  }
  for (int g = 0; g < l.n_groups; ++g) {
    launch_write_range(a, l, l.groups[g], l.groups[g + 1]);
    const int32_t e0 = g * l.group_events, e1 = std::min(a.n_events, (g + 1) * l.group_events);
    launch_cells_range(a, l, e0, e1, g + 1 == l.n_groups);
  }
}

// Launches only in the learned form (a.mlp set).
void step_cells_prefilter(const Arena &a, const Launch &l)
{
  if (a.mlp) {
    k_cells_prefilter<<<l.num_sms * kPrefilterBlocks, kPrefilterThreads, 0, l.stream>>>(a);
  }
}

void step_cells_scatter(const Arena &a, const Launch &l) { k_cells_scatter<<<blocks_for(l.num_sms * 8, l.tracklets / 32, kScatterThreads / 32), kScatterThreads, 0, l.stream>>>(a); }

void step_neighbour_reset(const Arena &a, const Launch &l)
{
  if (l.staged) {
    k_neighbour_reset<<<fixed_grid(l), l.block, 0, l.stream>>>(a);
  }
}

template <bool kWrite>
void step_neighbours(const Arena &a, const Launch &l) { k_neighbours<kWrite><<<blocks_for(fixed_grid(l), l.cells, l.block), l.block, 0, l.stream>>>(a); }

// Threads for about half of the cells of the largest event's largest layer (a layer of hits has about
// 1.3 cells per hit), so that a layer takes one or two rounds.
void step_levels(const Arena &a, const Launch &l)
{
  if (a.n_events <= 0) {
    return;
  }
  const LevelShape shape = level_shape(a.n_events, l.level_size, l.num_sms);
  if (shape.wide) {
    for (int layer = 1; layer < ITSU_CELL_LAYERS; ++layer) {
      k_levels_layer<<<event_grid(a, l), l.block, 0, l.stream>>>(a, layer);
    }
  } else if (shape.threads == 128) {
    launch_clusters(k_levels<128>, a.n_events, 1, 128, 0, l.stream, a);
  } else {
    launch_clusters(k_levels<512>, a.n_events, shape.ctas, 512, 0, l.stream, a);
  }
}

void step_roads(const Arena &a, const Launch &l)
{
  if (a.n_events > 0) {
    k_roads<<<event_grid(a, l), l.block, 0, l.stream>>>(a);
  } else {
    cudaMemsetAsync(a.road_seg, 0, sizeof(int32_t), l.stream);  // no road offsets but the end
  }
}

// The whole run, kernel by kernel, in launch order.
const KernelStep kSteps[] = {
    {"status_init", step_status_init, 0},                    // 0
    {"cluster_sort", step_cluster_sort, 0},                  // 1  (a)
    {"tracklets_count", step_tracklets_count, 0},            // 2  (b)
    {"tracklets_gate", step_tracklets_gate, kGateStep},      // 3  (learned form with the gate)
    {"scan_tracklets", step_scan<0>, 0},                     // 4
    {"tracklet_segments", step_tracklet_segments, 0},        // 5  (and a whole run's crowded clusters)
    {"tracklets_crowded", step_tracklets_crowded, kStagedStep},  // 6
    {"tracklets_write", step_tracklets_write, kUngroupedStep},  // 7
    {"cells_count", step_cells_count, kUngroupedStep},       // 8  (c)
    {"write_count_by_event_group", step_write_count_groups, kGroupedStep},  // 9 (tracklet write + cell count per group)
    {"cells_prefilter", step_cells_prefilter, kPairPrefilterStep},  // 10 (learned form with the pair prefilter)
    {"scan_cells", step_scan<1>, 0},                         // 11 (and the cell segments)
    {"cells_scatter", step_cells_scatter, 0},                // 12
    {"neighbour_reset", step_neighbour_reset, kStagedStep},  // 13 (d)
    {"neighbours_count", step_neighbours<false>, 0},         // 14
    {"scan_neighbours", step_scan<2>, 0},                    // 15
    {"neighbours_write", step_neighbours<true>, 0},          // 16
    {"levels", step_levels, 0},                              // 17
    {"scan_roads", step_scan<3>, 0},                         // 18 (e)
    {"roads_write", step_roads, 0},                          // 19
};
constexpr int kNumSteps = sizeof(kSteps) / sizeof(kSteps[0]);

void run_steps(int first, int last, const Arena &a, const Launch &l)
{
  for (int k = first; k <= last; ++k) {
    kSteps[k].launch(a, l);
  }
}

}  // namespace

// The clustering's launch for a run whose largest layer has max_segment clusters (any shape gives the
// same results). Small layers take small CTAs: the tables' set-up is most of their work. Layers of
// even size are split over clusters of 2 to 8 CTAs while that makes no more than 1024 of them (two to
// three waves at three CTAs on each of 148 SMs), so that the last wave is not nearly empty; where the
// sizes differ widely, the large ones only while the chip has room for all of them at once (296: two per
// SM).
SortShape sort_shape(int32_t n_events, int64_t n_clusters, int64_t max_segment)
{
  const int64_t segments = (int64_t)n_events * ITSU_LAYERS;
  SortShape s;
  s.threads = max_segment > 1024 ? 512 : (max_segment > 192 ? 256 : 64);
  s.ctas = 1;
  const int64_t most = 2 * n_clusters >= segments * max_segment ? 1024 : 296;
  while (max_segment > 1024 && s.ctas < 8 && 2 * s.ctas * segments <= most) {
    s.ctas *= 2;
  }
  return s;
}

// The level pass's launch for a run whose largest layer has as many cells as `size` clusters ordinarily
// give (Launch::level_size). A cluster of 8 CTAs has
// 4096 threads for an event's layer, and the cells of a layer grow with the square of its clusters: few
// events with large layers take a wide launch per layer instead. One event with layers of 9,450 clusters:
// 34 us in clusters, 28 wide; of 26,250: 126 and 38; of 52,500: 478 and 55. Four of 9,450: 37 and 38;
// eight of 12,600: 49 and 41; 16: 54 and 50; 32: 74 and 77.
constexpr int64_t kWideLevels = 10000;
LevelShape level_shape(int32_t n_events, int64_t size, int num_sms)
{
  LevelShape s;
  s.threads = size > 192 ? 512 : 128;
  s.ctas = 1;
  while (s.threads == 512 && s.ctas < 8 && 3 * size > 4 * 512 * s.ctas) {
    s.ctas *= 2;
  }
  s.wide = size > kWideLevels && 2 * (int64_t)n_events * s.ctas < 3 * num_sms;
  return s;
}

// Streamed host runs: appends the last run's roads and road offsets to the batch-wide output at
// event e0. The chunk's first road index is dst_off[e0], written by the previous chunk (or zeroed
// by the host); a chunk that overflowed or does not fit leaves its roads out and passes its base
// on, so the next chunk stays in bounds. The run's status goes to *snap for the host.
__global__ void k_append_roads(Arena a, itsu_road *dst, int32_t *dst_off, int32_t e0, int64_t cap, DevStatus *snap)
{
  const bool ok = !capacity_failed(a.status);
  int64_t base = dst_off[e0];
  base = base < 0 ? 0 : base;
  const int64_t total = ok ? a.status->total[kRoads] : 0;
  const bool fits = base + total <= cap;
  const int64_t tid = global_thread(), threads = grid_threads();
  if (ok && fits) {
    const int4 *from = reinterpret_cast<const int4 *>(a.roads);  // 32-byte records, two 16-byte words each
    int4 *to = reinterpret_cast<int4 *>(dst + base);
    for (int64_t r = tid; r < 2 * total; r += threads) {
      to[r] = from[r];
    }
    for (int64_t e = tid + 1; e <= a.n_events; e += threads) {
      dst_off[e0 + e] = (int32_t)(base + a.road_seg[e]);
    }
  } else {
    for (int64_t e = tid + 1; e <= a.n_events; e += threads) {
      dst_off[e0 + e] = (int32_t)base;
    }
  }
  if (tid == 0) {
    DevStatus st = *a.status;
    if (ok && !fits) {
      st.flags |= kFlagCapRoads;
    }
    *snap = st;
  }
}

__global__ void k_event_segments(Arena a, int32_t e, bool cells, bool neighbours, bool roads, EventSegments *out)
{
  const int k = threadIdx.x;
  if (k <= ITSU_TRACKLET_LAYERS) {
    out->ts[k] = a.trk_seg[(int64_t)e * ITSU_TRACKLET_LAYERS + k];
  }
  if (k <= ITSU_CELL_LAYERS) {
    const int32_t c = cells ? a.cell_seg[(int64_t)e * ITSU_CELL_LAYERS + k] : 0;
    out->cs[k] = c;
    out->nbo[k] = neighbours ? a.nb_off[c] : 0;
  }
  if (k < 2) {
    out->rs[k] = roads ? a.road_seg[e + k] : 0;
  }
}

void launch_event_segments(const Arena &a, int32_t e, bool cells, bool neighbours, bool roads, EventSegments *out, cudaStream_t stream)
{
  k_event_segments<<<1, 32, 0, stream>>>(a, e, cells, neighbours, roads, out);
}

void launch_append_roads(const Arena &a, const Launch &l, itsu_road *dst, int32_t *dst_off, int32_t e0, int64_t cap, DevStatus *snap)
{
  k_append_roads<<<l.num_sms * 2, 256, 0, l.stream>>>(a, dst, dst_off, e0, cap, snap);
}

const KernelStep *pipeline_steps(int *count)
{
  *count = kNumSteps;
  return kSteps;
}

void launch_status_init(const Arena &a, const Launch &l) { run_steps(0, 0, a, l); }
void launch_cluster_sort(const Arena &a, const Launch &l) { run_steps(1, 1, a, l); }
void launch_tracklets_count(const Arena &a, const Launch &l) { run_steps(2, 5, a, l); }

void launch_atan2f(const float *y, const float *x, float *out, int64_t n, int num_sms, cudaStream_t stream)
{
  if (n > 0) {
    k_atan2f<<<num_sms * 4, 256, 0, stream>>>(y, x, out, n);
  }
}
void launch_tracklets_write(const Arena &a, const Launch &l) { run_steps(6, 7, a, l); }
void launch_cells_count(const Arena &a, const Launch &l) { run_steps(8, 11, a, l); }
void launch_cells_write(const Arena &a, const Launch &l) { run_steps(12, 12, a, l); }
void launch_neighbours_count(const Arena &a, const Launch &l) { run_steps(13, 15, a, l); }
void launch_neighbours_write(const Arena &a, const Launch &l) { run_steps(16, 17, a, l); }
void launch_roads_count(const Arena &a, const Launch &l) { run_steps(18, 18, a, l); }
void launch_roads_write(const Arena &a, const Launch &l) { run_steps(19, 19, a, l); }

int kernels_per_run()
{
  int n = 0;
  for (const KernelStep &k : kSteps) {
    n += (k.learned_only == 0 || k.learned_only == kUngroupedStep) ? 1 : 0;
  }
  return n;
}

}  // namespace itsu
