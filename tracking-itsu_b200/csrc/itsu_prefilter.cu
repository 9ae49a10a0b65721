// itsu_prefilter.cu - the learned prefilter's training-side kernels: sample export, scoring,
// minibatch gradients and the Adam step.
//
// Inference lives in the cell stage (k_cells_prefilter, itsu_kernels.cu: each cell entry's
// features, the three layers and the threshold in one pass, no feature rows in memory); the
// scorer here runs the same device code (pair_features, mlp_logits_warp) on exported feature
// rows, so that the two give the same logit for the same pair. Training is binary cross-entropy on the sigmoid output with
// the forward pass exactly as inference computes it (BF16 inputs, weights and activations, FP32
// accumulation) and the backward pass on the tensor cores too: the gradients with respect to the
// pre-activations are rounded to BF16 for the three backward MMAs (dW2, dh1, dW1), accumulated in
// FP32, and applied to FP32 master weights (the BF16 rounding of the forward pass is passed
// straight through).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "itsu_device.cuh"
#include "itsu_internal.h"
#include "itsu_mlp.cuh"

namespace itsu {
namespace {

constexpr int kTrainWarps = 4;
constexpr int kTrainSamples = 16 * kTrainWarps;  // a block's tile
constexpr int kMaxGradBlocks = 2 * 148;          // two per SM of a B200; each leaves a gradient partial

__device__ __forceinline__ uint64_t splitmix64(uint64_t x)
{
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// ---- publish: FP32 master -> device model ----

// The FP32 master of an 8 -> H -> H -> 1 network (itsu_prefilter_model / itsu_gate_model): the
// trainable parameters in MlpShape<H> order, then mean[8], inv_std[8] and the logit threshold.
template <int H>
__device__ __forceinline__ void publish_param(MlpDeviceT<H> *model, int i, float w)
{
  using S = MlpShape<H>;
  if (i < S::kOffB1) {
    model->w1[i / kMlpIn][i % kMlpIn] = __float2bfloat16_rn(w);
  } else if (i < S::kOffW2) {
    model->b1[i - S::kOffB1] = w;
  } else if (i < S::kOffB2) {
    model->w2[(i - S::kOffW2) / H][(i - S::kOffW2) % H] = __float2bfloat16_rn(w);
  } else if (i < S::kOffW3) {
    model->b2[i - S::kOffB2] = w;
  } else if (i < S::kOffB3) {
    model->w3[i - S::kOffW3] = __float2bfloat16_rn(w);
  } else {
    model->b3 = w;
  }
}

// window: the gate's per-layer |dphi| window in the master (null for the pair prefilter: pi).
template <int H>
__global__ void k_mlp_publish(const float *master, const float *window, const float *dz_window, const int32_t *mlp_layers,
                              MlpDeviceT<H> *model)
{
  constexpr int P = MlpShape<H>::kParams;
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    publish_param<H>(model, i, master[i]);
  }
  for (int i = threadIdx.x; i < kMlpIn; i += blockDim.x) {
    model->mean[i] = master[P + i];
    model->inv_std[i] = master[P + kMlpIn + i];
  }
  for (int i = threadIdx.x; i < 6; i += blockDim.x) {
    model->window[i] = window ? window[i] : 3.14159265358979323846f;
    model->dz_window[i] = dz_window ? dz_window[i] : HUGE_VALF;
  }
  if (threadIdx.x == 0) {
    model->threshold = master[P + 2 * kMlpIn];
    model->mlp_layers = mlp_layers ? (uint32_t)*mlp_layers : 0x3fu;
  }
}

// ---- export: one sample per cell, road membership and road keys ----

__global__ void k_export_cells(Arena a, itsu_prefilter_samples out)
{
  const int64_t n = a.status->total[kCells];
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
    if (out.labels) {
      out.labels[c] = 0;
    }
    if (!out.features) {
      continue;
    }
    const int sid = a.cell_seg_id[c];
    const int e = sid / ITSU_CELL_LAYERS, layer = sid % ITSU_CELL_LAYERS;
    const itsu_cell cell = a.cells[c];
    const int32_t *ts = a.trk_seg + e * ITSU_TRACKLET_LAYERS;
    const int32_t *lo = a.layer_off + e * ITSU_LAYERS;
    const itsu_tracklet t1 = a.tracklets[ts[layer] + cell.first_tracklet];
    const itsu_tracklet t2 = a.tracklets[ts[layer + 1] + cell.second_tracklet];
    const float4 c1 = a.xyzr[lo[layer] + cell.first_cluster];
    const float4 c2 = a.xyzr[lo[layer + 1] + cell.second_cluster];
    const float4 c3 = a.xyzr[lo[layer + 2] + cell.third_cluster];
    const float vx = a.vtx[3 * e], vy = a.vtx[3 * e + 1], vz = a.vtx[3 * e + 2];
    float3 normal;
    float curvature, dca;
    cell_geometry(layer, c1, c2, c3, vx, vy, normal, curvature, dca);
    float f[kMlpIn];
    pair_features(layer, t1.tan_lambda, t1.phi, t2.tan_lambda, t2.phi, c1, c2, c3, vx, vy, vz, dca, f);
    float4 *dst = reinterpret_cast<float4 *>(out.features + c * kMlpIn);
    dst[0] = make_float4(f[0], f[1], f[2], f[3]);
    dst[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
}

__global__ void k_export_roads(Arena a, itsu_prefilter_samples out)
{
  const int64_t n = a.status->total[kRoads];
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    // event of the road: last e with road_seg[e] <= r
    int lo_e = 0, hi_e = a.n_events - 1;
    while (lo_e < hi_e) {
      const int mid = (lo_e + hi_e + 1) >> 1;
      if (a.road_seg[mid] <= r) {
        lo_e = mid;
      } else {
        hi_e = mid - 1;
      }
    }
    const int e = lo_e;
    const itsu_road road = a.roads[r];
    const int32_t *cs = a.cell_seg + e * ITSU_CELL_LAYERS;
    int32_t key[ITSU_LAYERS];
    for (int l = 0; l < ITSU_CELL_LAYERS; ++l) {
      const int64_t gc = cs[l] + road.cell_ids[l];
      if (out.labels) {
        out.labels[gc] = 1;
      }
      if (out.road_cells) {
        out.road_cells[r * ITSU_CELL_LAYERS + l] = (int32_t)gc;
      }
      const itsu_cell cell = a.cells[gc];
      if (l == 0) {
        key[0] = cell.first_cluster;
        key[1] = cell.second_cluster;
      }
      key[l + 2] = cell.third_cluster;
    }
    if (out.road_keys) {
      int32_t *k = out.road_keys + r * 8;
      k[0] = e;
      for (int l = 0; l < ITSU_LAYERS; ++l) {
        k[l + 1] = key[l];
      }
    }
    if (out.road_fake) {
      out.road_fake[r] = road.is_fake;
    }
  }
}

// ---- gate export: one sample per tracklet, on-road labels ----

__global__ void k_export_tracklets(Arena a, itsu_gate_samples out)
{
  const int64_t n = a.status->total[kTracklets];
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    if (out.labels) {
      out.labels[k] = 0;
    }
    if (!out.features) {
      continue;
    }
    const int sid = tracklet_segment(a, k);
    const int e = sid / ITSU_TRACKLET_LAYERS, layer = sid % ITSU_TRACKLET_LAYERS;
    const itsu_tracklet t = a.tracklets[k];
    const int32_t *lo = a.layer_off + e * ITSU_LAYERS;
    const int64_t i1 = lo[layer] + t.first_cluster, i2 = lo[layer + 1] + t.second_cluster;
    float f[kMlpIn];
    tracklet_features(layer, a.xyzr[i1], a.phi[i1], a.xyzr[i2], a.phi[i2], a.vtx[3 * e], a.vtx[3 * e + 1], a.vtx[3 * e + 2], f);
    float4 *dst = reinterpret_cast<float4 *>(out.features + k * kMlpIn);
    dst[0] = make_float4(f[0], f[1], f[2], f[3]);
    dst[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
}

// Marks the two tracklets of every cell of every road (after k_export_tracklets cleared them) and
// lists each road's tracklets, layers 0..5 (-1 where the road has no cell).
__global__ void k_export_tracklet_labels(Arena a, itsu_gate_samples out)
{
  const int64_t n = a.status->total[kRoads];
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    int lo_e = 0, hi_e = a.n_events - 1;  // the road's event: last e with road_seg[e] <= r
    while (lo_e < hi_e) {
      const int mid = (lo_e + hi_e + 1) >> 1;
      if (a.road_seg[mid] <= r) {
        lo_e = mid;
      } else {
        hi_e = mid - 1;
      }
    }
    const itsu_road road = a.roads[r];
    const int32_t *cs = a.cell_seg + lo_e * ITSU_CELL_LAYERS;
    const int32_t *ts = a.trk_seg + lo_e * ITSU_TRACKLET_LAYERS;
    int32_t rows[ITSU_TRACKLET_LAYERS];
    for (int l = 0; l < ITSU_TRACKLET_LAYERS; ++l) {
      rows[l] = -1;
    }
    for (int l = 0; l < ITSU_CELL_LAYERS; ++l) {
      if (road.cell_ids[l] < 0) {
        continue;
      }
      const itsu_cell cell = a.cells[cs[l] + road.cell_ids[l]];
      rows[l] = ts[l] + cell.first_tracklet;
      rows[l + 1] = ts[l + 1] + cell.second_tracklet;
    }
    for (int l = 0; l < ITSU_TRACKLET_LAYERS; ++l) {
      if (out.labels && rows[l] >= 0) {
        out.labels[rows[l]] = 1;
      }
      if (out.road_tracklets) {
        out.road_tracklets[r * ITSU_TRACKLET_LAYERS + l] = rows[l];
      }
    }
  }
}

// ---- scoring ----

constexpr int kScoreThreads = 256;

template <int H, bool kRelu>
__global__ void __launch_bounds__(kScoreThreads) k_mlp_score(const MlpDeviceT<H> *model, const float *features, int64_t n,
                                                            float *logits)
{
  __shared__ MlpSmemT<H> mlp;
  __shared__ __align__(16) __nv_bfloat16 rows[kScoreThreads / 32][32][kRowPitch];
  load_mlp(mlp, *model);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tiles = (n + 31) / 32;
  for (int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp; tile < tiles; tile += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    const int64_t row = tile * 32 + lane;
    float f[kMlpIn];
    for (int k = 0; k < kMlpIn; ++k) {
      f[k] = row < n ? features[row * kMlpIn + k] : mlp.mean[k];
    }
    feature_row(mlp.mean, mlp.inv_std, f, rows[warp][lane]);
    __syncwarp();
    const float logit = mlp_logits_warp<H, kRelu>(mlp, rows[warp]);
    if (row < n) {
      logits[row] = logit;
    }
    __syncwarp();
  }
}

// ---- training: minibatch gradient ----

// A block's tile of the training pass of an 8 -> H -> H -> 1 network, [sample][unit], as the weight
// gradients' operands, and what each warp's samples add to the sums over samples.
template <int H>
struct __align__(16) TrainBlock {
  static constexpr int kPitch = MlpShape<H>::kHidPitch;
  MlpSmemT<H> mlp;
  __align__(16) __nv_bfloat16 x[kTrainSamples][kRowPitch];  // standardised inputs
  __nv_bfloat16 h1[kTrainSamples][kPitch];                  // layer-1 activations
  __nv_bfloat16 d2[kTrainSamples][kPitch];                  // dL/da2
  __nv_bfloat16 d1[kTrainSamples][kPitch];                  // dL/da1
  float unit[kTrainWarps][3][H];                            // dL/dW3, dL/db2, dL/db1
  float b3[kTrainWarps];
};

// Gradient of the loss over a batch. A block takes tiles of 64 samples. A warp has 16 of them, as the
// rows of one MMA, and keeps their forward and backward pass in registers, one layer's output
// fragments being the next one's operand; then the block's warps share out the rows of dL/dW2 and
// dL/dW1, contractions over all 64 samples, whose accumulators stay in registers over the block's
// tiles, like the sums over samples (biases, W3, loss). Each block writes its partial gradient.
// Bound by the latency of one tile's chain (a batch of 8192 is 128 tiles, one per SM) and of the
// network's load: 13 us per batch of 8192, 0.075 ms per 262,144 samples; 38 us and 0.79 ms with 32
// samples per warp passed through shared memory and gradients summed by shared-memory atomics.
template <int H, bool kRelu>
__global__ void __launch_bounds__(kTrainWarps * 32, 2) k_mlp_gradient(const MlpDeviceT<H> *model, const float *features,
                                                                      const uint8_t *labels, int64_t n, int32_t batch,
                                                                      int32_t sequential, uint64_t seed, int64_t step,
                                                                      float pos_weight, float *grad_partials, float *loss)
{
  using S = MlpShape<H>;
  constexpr int NT = H / 8, KT = H / 16;
  constexpr int kRowTiles = (KT + kTrainWarps - 1) / kTrainWarps;  // of dL/dW2 and dL/dW1 per warp
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainBlock<H> &B = *reinterpret_cast<TrainBlock<H> *>(smem_raw);
  const MlpSmemT<H> &M = B.mlp;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  // half a sample of the warp's in a tile, and its label: two lanes per sample
  float4 half_row = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float y = 0.0f;
  auto fetch = [&](int64_t tile) {
    const int64_t k = tile * kTrainSamples + warp * 16 + (lane >> 1);
    if (k < batch) {
      const int64_t idx = sequential ? k : (int64_t)(splitmix64(seed + (uint64_t)step * 0x632BE59BD9B4E019ull + (uint64_t)k) % (uint64_t)n);
      half_row = reinterpret_cast<const float4 *>(features + idx * kMlpIn)[lane & 1];
      y = labels[idx] ? 1.0f : 0.0f;
    }
  };
  fetch(blockIdx.x);  // under way while the network is loaded
  load_mlp(B.mlp, *model);
  __syncthreads();
  const int mq = lane >> 3, mr = lane & 7;  // the matrix and row whose address the lane gives to ldmatrix_t
  const int r0 = warp * 16 + g, r1 = r0 + 8;
  const float inv_batch = 1.0f / (float)batch;
  float dw2[kRowTiles][NT][4] = {}, dw1[kRowTiles][4] = {};
  float dw3[NT][2] = {}, db2[NT][2] = {}, db1[NT][2] = {};  // of columns nt * 8 + 2t, + 1: rows r0 and r1 of every tile
  float db3 = 0.0f, loss_sum = 0.0f;
  const int64_t tiles = ((int64_t)batch + kTrainSamples - 1) / kTrainSamples;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    // 1. the warp's samples as MMA rows
    const bool valid = tile * kTrainSamples + warp * 16 + (lane >> 1) < batch;
    {
      const int half = lane & 1;
      const float4 u = half_row;
      const float *mean = M.mean + 4 * half, *inv_std = M.inv_std + 4 * half;
      uint2 *const row = reinterpret_cast<uint2 *>(B.x[warp * 16 + (lane >> 1)]);
      row[half] = valid ? make_uint2(pack_bf16((u.x - mean[0]) * inv_std[0], (u.y - mean[1]) * inv_std[1]),
                                     pack_bf16((u.z - mean[2]) * inv_std[2], (u.w - mean[3]) * inv_std[3]))
                        : make_uint2(0, 0);
      row[2 + half] = make_uint2(0, 0);
    }
    const float weight = valid ? (y > 0.0f ? pos_weight : 1.0f) : 0.0f;
    const float y0 = __shfl_sync(0xffffffffu, y, 2 * g), y1 = __shfl_sync(0xffffffffu, y, 2 * g + 16);
    const float weight0 = __shfl_sync(0xffffffffu, weight, 2 * g), weight1 = __shfl_sync(0xffffffffu, weight, 2 * g + 16);
    __syncwarp();
    // 2. forward, keeping the activations' derivatives
    uint32_t a[4], h1[KT][4], h2[KT][4];
    float e1[NT][4], e2[NT][4];
    a[0] = ld32(&B.x[r0][2 * t]);
    a[1] = ld32(&B.x[r1][2 * t]);
    a[2] = ld32(&B.x[r0][2 * t + 8]);
    a[3] = ld32(&B.x[r1][2 * t + 8]);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int col = nt * 8 + 2 * t;
      float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      mma_bf16(c, a, ld32(&M.w1[nt * 8 + g][2 * t]), ld32(&M.w1[nt * 8 + g][2 * t + 8]));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        c[q] += M.b1[col + (q & 1)];
        e1[nt][q] = act_grad<kRelu>(c[q]);
        c[q] = act<kRelu>(c[q]);
      }
      const uint32_t top = pack_bf16(c[0], c[1]), bottom = pack_bf16(c[2], c[3]);
      h1[nt >> 1][(nt & 1) * 2 + 0] = top;
      h1[nt >> 1][(nt & 1) * 2 + 1] = bottom;
      *reinterpret_cast<uint32_t *>(&B.h1[r0][col]) = top;
      *reinterpret_cast<uint32_t *>(&B.h1[r1][col]) = bottom;
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int col = nt * 8 + 2 * t;
      float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        mma_bf16(c, h1[kk], ld32(&M.w2[nt * 8 + g][16 * kk + 2 * t]), ld32(&M.w2[nt * 8 + g][16 * kk + 2 * t + 8]));
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        c[q] += M.b2[col + (q & 1)];
        e2[nt][q] = act_grad<kRelu>(c[q]);
        c[q] = act<kRelu>(c[q]);
      }
      h2[nt >> 1][(nt & 1) * 2 + 0] = pack_bf16(c[0], c[1]);
      h2[nt >> 1][(nt & 1) * 2 + 1] = pack_bf16(c[2], c[3]);
    }
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      mma_bf16(o, h2[kk], ld32(&M.w3[g][16 * kk + 2 * t]), ld32(&M.w3[g][16 * kk + 2 * t + 8]));
    }
    // 3. loss and dL/dz: weighted binary cross-entropy of sigmoid(z), averaged over the batch; the
    // logits of rows r0 and r1 stand in the quad's first lane
    const float z0 = __shfl_sync(0xffffffffu, o[0] + M.b3, lane & ~3), z1 = __shfl_sync(0xffffffffu, o[2] + M.b3, lane & ~3);
    const float dz0 = weight0 * (1.0f / (1.0f + expf(-z0)) - y0) * inv_batch, dz1 = weight1 * (1.0f / (1.0f + expf(-z1)) - y1) * inv_batch;
    if (t == 0) {
      loss_sum += weight0 * (fmaxf(z0, 0.0f) - z0 * y0 + log1pf(expf(-fabsf(z0)))) * inv_batch;
      loss_sum += weight1 * (fmaxf(z1, 0.0f) - z1 * y1 + log1pf(expf(-fabsf(z1)))) * inv_batch;
      db3 += dz0 + dz1;
    }
    // 4. dL/dW3, dL/da2
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int col = nt * 8 + 2 * t;
      const __nv_bfloat162 top = *reinterpret_cast<const __nv_bfloat162 *>(&h2[nt >> 1][(nt & 1) * 2 + 0]);
      const __nv_bfloat162 bottom = *reinterpret_cast<const __nv_bfloat162 *>(&h2[nt >> 1][(nt & 1) * 2 + 1]);
      dw3[nt][0] += dz0 * __bfloat162float(top.x) + dz1 * __bfloat162float(bottom.x);
      dw3[nt][1] += dz0 * __bfloat162float(top.y) + dz1 * __bfloat162float(bottom.y);
      const float w0 = __bfloat162float(M.w3[0][col]), w1 = __bfloat162float(M.w3[0][col + 1]);
      const float d0 = dz0 * w0 * e2[nt][0], d1 = dz0 * w1 * e2[nt][1], d2 = dz1 * w0 * e2[nt][2], d3 = dz1 * w1 * e2[nt][3];
      db2[nt][0] += d0 + d2;
      db2[nt][1] += d1 + d3;
      const uint32_t d_top = pack_bf16(d0, d1), d_bottom = pack_bf16(d2, d3);
      h2[nt >> 1][(nt & 1) * 2 + 0] = d_top;  // from here on dL/da2
      h2[nt >> 1][(nt & 1) * 2 + 1] = d_bottom;
      *reinterpret_cast<uint32_t *>(&B.d2[r0][col]) = d_top;
      *reinterpret_cast<uint32_t *>(&B.d2[r1][col]) = d_bottom;
    }
    // 5. dL/da1 = (dL/da2 W2) * act'(a1): [16 s x H j] x [H j x H i]
#pragma unroll
    for (int nt = 0; nt < NT; nt += 2) {
      float c[2][4] = {};
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        uint32_t w[4];
        ldmatrix_t(w, &M.w2[16 * kk + (mq & 1) * 8 + mr][(nt + (mq >> 1)) * 8]);
        mma_bf16(c[0], h2[kk], w[0], w[1]);
        mma_bf16(c[1], h2[kk], w[2], w[3]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int col = (nt + h) * 8 + 2 * t;
        const float d0 = c[h][0] * e1[nt + h][0], d1 = c[h][1] * e1[nt + h][1], d2 = c[h][2] * e1[nt + h][2], d3 = c[h][3] * e1[nt + h][3];
        db1[nt + h][0] += d0 + d2;
        db1[nt + h][1] += d1 + d3;
        *reinterpret_cast<uint32_t *>(&B.d1[r0][col]) = pack_bf16(d0, d1);
        *reinterpret_cast<uint32_t *>(&B.d1[r1][col]) = pack_bf16(d2, d3);
      }
    }
    __syncthreads();
    // 6. dL/dW2 = dL/da2^T h1: [H j x 64 s] x [64 s x H i], dL/dW1 = dL/da1^T x: [H i x 64 s] x [64 s x 8 f]
#pragma unroll
    for (int m = 0; m < kRowTiles; ++m) {
      const int mt = warp + m * kTrainWarps;
      if (mt < KT) {
#pragma unroll
        for (int kk = 0; kk < kTrainSamples / 16; ++kk) {
          uint32_t d[4], b[4];
          ldmatrix_t(d, &B.d2[16 * kk + (mq >> 1) * 8 + mr][16 * mt + (mq & 1) * 8]);
#pragma unroll
          for (int nt = 0; nt < NT; nt += 2) {
            ldmatrix_t(b, &B.h1[16 * kk + (mq & 1) * 8 + mr][(nt + (mq >> 1)) * 8]);
            mma_bf16(dw2[m][nt], d, b[0], b[1]);
            mma_bf16(dw2[m][nt + 1], d, b[2], b[3]);
          }
          ldmatrix_t(d, &B.d1[16 * kk + (mq >> 1) * 8 + mr][16 * mt + (mq & 1) * 8]);
          ldmatrix_t(b, &B.x[16 * kk + (mq & 1) * 8 + mr][0]);
          mma_bf16(dw1[m], d, b[0], b[1]);
        }
      }
    }
    fetch(tile + gridDim.x);
    __syncthreads();  // the tile is refilled
  }
  // The block's partial gradient.
  float *out = grad_partials + (int64_t)blockIdx.x * S::kParams;
#pragma unroll
  for (int m = 0; m < kRowTiles; ++m) {
    const int mt = warp + m * kTrainWarps;
    if (mt < KT) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = 16 * mt + g + 8 * h;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          out[S::kOffW2 + row * H + nt * 8 + 2 * t] = dw2[m][nt][2 * h];
          out[S::kOffW2 + row * H + nt * 8 + 2 * t + 1] = dw2[m][nt][2 * h + 1];
        }
        out[S::kOffW1 + row * kMlpIn + 2 * t] = dw1[m][2 * h];
        out[S::kOffW1 + row * kMlpIn + 2 * t + 1] = dw1[m][2 * h + 1];
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float s3 = dw3[nt][q], s2 = db2[nt][q], s1 = db1[nt][q];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        s3 += __shfl_xor_sync(0xffffffffu, s3, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      }
      if (g == 0) {
        const int col = nt * 8 + 2 * t + q;
        B.unit[warp][0][col] = s3;
        B.unit[warp][1][col] = s2;
        B.unit[warp][2][col] = s1;
      }
    }
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {  // the quads' first lanes
    db3 += __shfl_xor_sync(0xffffffffu, db3, o);
    loss_sum += __shfl_xor_sync(0xffffffffu, loss_sum, o);
  }
  if (lane == 0) {
    B.b3[warp] = db3;
    atomicAdd(loss, loss_sum);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * H + 1; i += blockDim.x) {
    float sum = 0.0f;
    for (int w = 0; w < kTrainWarps; ++w) {
      sum += i < 3 * H ? B.unit[w][i / H][i % H] : B.b3[w];
    }
    const int to = i < H ? S::kOffW3 + i : (i < 2 * H ? S::kOffB2 + i - H : (i < 3 * H ? S::kOffB1 + i - 2 * H : S::kOffB3));
    out[to] = sum;
  }
}

// A parameter's partials, one of kSumSlices threads per slice of the blocks: the sum is in the first
// slice's thread. 32 parameters per block of threads, so that a warp reads consecutive ones.
constexpr int kSumSlices = 8;

template <class T, int kParams>
__device__ __forceinline__ T sum_partials(const float *grad_partials, int blocks, int i, T (*part)[32])
{
  const int slice = threadIdx.x / 32, at = threadIdx.x % 32;
  T sum = 0;
  if (i < kParams) {
#pragma unroll 16
    for (int b = slice; b < blocks; b += kSumSlices) {
      sum += grad_partials[(int64_t)b * kParams + i];
    }
  }
  part[slice][at] = sum;
  __syncthreads();
  if (slice == 0) {
    for (int s = 1; s < kSumSlices; ++s) {
      sum += part[s][at];
    }
  }
  return sum;
}

template <int H>
__global__ void __launch_bounds__(32 * kSumSlices) k_mlp_gradient_sum(const float *grad_partials, int blocks, float *grad)
{
  __shared__ double part[kSumSlices][32];
  const int i = blockIdx.x * 32 + threadIdx.x % 32;
  const double sum = sum_partials<double, MlpShape<H>::kParams>(grad_partials, blocks, i, part);
  if (threadIdx.x < 32 && i < MlpShape<H>::kParams) {
    grad[i] = (float)sum;
  }
}

// ---- Adam ----

// One step on the sum of the partials (32 parameters per block; 4 us, 6 with a thread per parameter
// that adds up all partials).
template <int H>
__global__ void __launch_bounds__(32 * kSumSlices) k_mlp_adam(float *master, const float *grad_partials, int blocks, float *m, float *v,
                                                              float lr, float beta1, float beta2, float eps, float weight_decay,
                                                              float bias1, float bias2, MlpDeviceT<H> *model)
{
  using S = MlpShape<H>;
  __shared__ float part[kSumSlices][32];
  const int i = blockIdx.x * 32 + threadIdx.x % 32;
  const bool own = threadIdx.x < 32 && i < S::kParams;
  float m0 = 0.0f, v0 = 0.0f, w = 0.0f;  // under way with the partials
  if (own) {
    m0 = m[i];
    v0 = v[i];
    w = master[i];
  }
  const float gsum = sum_partials<float, S::kParams>(grad_partials, blocks, i, part);
  if (!own) {
    return;
  }
  const float mm = beta1 * m0 + (1.0f - beta1) * gsum;
  const float vv = beta2 * v0 + (1.0f - beta2) * gsum * gsum;
  m[i] = mm;
  v[i] = vv;
  const bool is_weight = i < S::kOffB1 || (i >= S::kOffW2 && i < S::kOffB2) || (i >= S::kOffW3 && i < S::kOffB3);
  if (is_weight) {
    w -= lr * weight_decay * w;
  }
  w -= lr * (mm / bias1) / (sqrtf(vv / bias2) + eps);
  master[i] = w;
  publish_param<H>(model, i, w);
}

int gradient_blocks(int32_t batch)
{
  const int64_t blocks = ((int64_t)batch + kTrainSamples - 1) / kTrainSamples;
  return (int)(blocks < kMaxGradBlocks ? (blocks > 0 ? blocks : 1) : kMaxGradBlocks);
}

}  // namespace

namespace {

template <int H, bool kRelu>
void score_net(const MlpDeviceT<H> *model, const float *features, int64_t n, float *logits, int num_sms, cudaStream_t stream)
{
  const int64_t tiles = (n + 31) / 32;
  int64_t blocks = (tiles + kScoreThreads / 32 - 1) / (kScoreThreads / 32);
  if (blocks > (int64_t)num_sms * 8) {
    blocks = (int64_t)num_sms * 8;
  }
  if (blocks > 0) {
    k_mlp_score<H, kRelu><<<(unsigned)blocks, kScoreThreads, 0, stream>>>(model, features, n, logits);
  }
}

template <int H, bool kRelu>
void gradient_net(const MlpDeviceT<H> *model, const float *features, const uint8_t *labels, int64_t n, int32_t batch, bool sequential,
                  uint64_t seed, int64_t step, float pos_weight, float *grad_partials, float *loss, cudaStream_t stream)
{
  static_assert(sizeof(TrainBlock<H>) <= 48 * 1024, "within the default limit");
  k_mlp_gradient<H, kRelu><<<gradient_blocks(batch), kTrainWarps * 32, sizeof(TrainBlock<H>), stream>>>(
      model, features, labels, n, batch, sequential ? 1 : 0, seed, step, pos_weight, grad_partials, loss);
}

}  // namespace

static_assert(sizeof(itsu_prefilter_model) == sizeof(float) * (kMlpParams + 2 * kMlpIn + 1), "pair model layout");
static_assert(sizeof(itsu_gate_model) == sizeof(float) * (kGateParams + 2 * kMlpIn + 1 + 2 * ITSU_TRACKLET_LAYERS + 1), "gate model layout");

size_t mlp_device_bytes() { return sizeof(MlpDevice); }
size_t gate_device_bytes() { return sizeof(GateDevice); }
int mlp_gradient_blocks(int32_t batch) { return gradient_blocks(batch); }

void launch_mlp_gradient_sum(const float *grad_partials, int blocks, int params, float *grad, cudaStream_t stream)
{
  if (params == kMlpParams) {
    k_mlp_gradient_sum<kMlpHidden><<<(kMlpParams + 31) / 32, 32 * kSumSlices, 0, stream>>>(grad_partials, blocks, grad);
  } else {
    k_mlp_gradient_sum<kGateHidden><<<(kGateParams + 31) / 32, 32 * kSumSlices, 0, stream>>>(grad_partials, blocks, grad);
  }
}

void launch_mlp_publish(const itsu_prefilter_model *master, MlpDevice *model, cudaStream_t stream)
{
  k_mlp_publish<kMlpHidden><<<1, 512, 0, stream>>>(&master->w1[0][0], nullptr, nullptr, nullptr, model);
}

void launch_mlp_publish(const itsu_gate_model *master, GateDevice *model, cudaStream_t stream)
{
  k_mlp_publish<kGateHidden><<<1, 512, 0, stream>>>(&master->w1[0][0], &master->dphi_window[0], &master->dz_window[0],
                                                     &master->mlp_layers, model);
}

void launch_prefilter_export(const Arena &a, const itsu_prefilter_samples &out, int num_sms, cudaStream_t stream)
{
  k_export_cells<<<num_sms * 8, 256, 0, stream>>>(a, out);
  k_export_roads<<<num_sms * 4, 256, 0, stream>>>(a, out);
}

void launch_gate_export(const Arena &a, const itsu_gate_samples &out, int num_sms, cudaStream_t stream)
{
  k_export_tracklets<<<num_sms * 8, 256, 0, stream>>>(a, out);
  if (out.labels || out.road_tracklets) {
    k_export_tracklet_labels<<<num_sms * 4, 256, 0, stream>>>(a, out);
  }
}

void launch_mlp_score(const MlpDevice *model, const float *features, int64_t n, float *logits, int num_sms, cudaStream_t stream)
{
  score_net<kMlpHidden, false>(model, features, n, logits, num_sms, stream);
}

void launch_mlp_score(const GateDevice *model, const float *features, int64_t n, float *logits, int num_sms, cudaStream_t stream)
{
  score_net<kGateHidden, true>(model, features, n, logits, num_sms, stream);
}

void launch_mlp_gradient(const MlpDevice *model, const float *features, const uint8_t *labels, int64_t n, int32_t batch,
                         bool sequential, uint64_t seed, int64_t step, float pos_weight, float *grad_partials, float *loss,
                         cudaStream_t stream)
{
  gradient_net<kMlpHidden, false>(model, features, labels, n, batch, sequential, seed, step, pos_weight, grad_partials, loss, stream);
}

void launch_mlp_gradient(const GateDevice *model, const float *features, const uint8_t *labels, int64_t n, int32_t batch,
                         bool sequential, uint64_t seed, int64_t step, float pos_weight, float *grad_partials, float *loss,
                         cudaStream_t stream)
{
  gradient_net<kGateHidden, true>(model, features, labels, n, batch, sequential, seed, step, pos_weight, grad_partials, loss, stream);
}

void launch_mlp_adam(itsu_prefilter_model *master, const float *grad_partials, int blocks, float *m, float *v, float lr,
                     float beta1, float beta2, float eps, float weight_decay, float bias1, float bias2, MlpDevice *model,
                     cudaStream_t stream)
{
  k_mlp_adam<kMlpHidden><<<(kMlpParams + 31) / 32, 32 * kSumSlices, 0, stream>>>(&master->w1[0][0], grad_partials, blocks, m, v, lr,
                                                                                 beta1, beta2, eps, weight_decay, bias1, bias2, model);
}

void launch_mlp_adam(itsu_gate_model *master, const float *grad_partials, int blocks, float *m, float *v, float lr, float beta1,
                     float beta2, float eps, float weight_decay, float bias1, float bias2, GateDevice *model, cudaStream_t stream)
{
  k_mlp_adam<kGateHidden><<<(kGateParams + 31) / 32, 32 * kSumSlices, 0, stream>>>(&master->w1[0][0], grad_partials, blocks, m, v, lr,
                                                                                   beta1, beta2, eps, weight_decay, bias1, bias2, model);
}

}  // namespace itsu
