// Training of the learned subgrid closure on the GPU (include/psl.h, psl_sgs_trainer_*):
// training samples filtered from fine-grid runs of this solver, the closure's forward and
// backward passes, a deterministic cross-block gradient reduction and Adam.
//
// Samples.  A fine periodic box of 2M physical cells per axis (grid 2M+1 x 2M+1 x 2M: the
// x and y faces are the duplicated layers of applyBCPeriodicX/Y, periodicXY.h:11-101; z
// wraps through the periodic shift) is box-filtered 2x to M^3 coarse cells:
//   * the 8 children's populations are averaged and rescaled fine -> coarse
//     (gridRefinementFunctions.h:6-281, the transfer the solver's own restriction uses);
//     the features are those the coarse solver's update kernel would compute from them;
//   * the target is the least-squares eddy viscosity of the filtered field,
//       nu_t* = max(0, -tau^d : S / (2 S : S)),
//     tau_ij = <u_i u_j> - <u>_i <u>_j over the 8 children, S the strain rate of the
//     filtered velocity (central differences, periodic), in coarse lattice units.
//
// Gradients.  The loss is the mean over a batch of (softplus(z) - nu_t*/out_scale)^2.  Each
// warp takes tiles of 32 samples through the forward pass, the backward pass and the weight
// gradients as register-tiled matrix products (grad_kernel); blocks write partial gradients
// that a second kernel sums in a fixed order in FP64, in training together with the Adam
// update.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "psl.h"
#include "psl_internal.h"
#include "psl_kernels.cuh"
#include "psl_launch.cuh"
#include "psl_mlp.cuh"

using namespace psl;

namespace {

// flat parameter vector: w1 [32][10], b1 [32], w2 [32][32], b2 [32], w3 [32], b3, then the
// normalisation (in_shift [10], in_scale [10], out_scale), which training does not change
constexpr int kW1 = 0, kB1 = 320, kW2 = 352, kB2 = 1376, kW3 = 1408, kB3 = 1440, kTrainable = 1441;
constexpr int kShift = 1441, kScale = 1451, kOutScale = 1461, kParams = 1462;
constexpr int kMaxGradWarps = 14;
constexpr int kGradBlocks = 148;  // one block per SM (159 KB of shared memory at 14 warps)
// Tiles a warp adds up in FP32 before FP64 takes over: 128 samples a chain.  Larger batches run
// in pieces of kPieceSamples, whose sums are added in FP64.  One chain over all of a batch of 2^22
// equal samples (2,048 products each) was off by 2.9e-5 of the gradient.
constexpr int kMaxTilesPerWarp = 4;
constexpr int kTile = 32;         // samples per warp tile
constexpr long long kPieceSamples = (long long)kGradBlocks * kMaxGradWarps * kMaxTilesPerWarp * kTile;
constexpr int kLd = 36;           // floats per row of 32 samples: consecutive rows 4 banks apart

int fail(int code, const std::string& msg) {
  psl_detail_set_last_error(msg);
  return code;
}

#define TRAIN_CUDA(expr)                                                                               \
  do {                                                                                                 \
    cudaError_t e_ = (expr);                                                                           \
    if (e_ != cudaSuccess) return fail(PSL_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
  } while (0)

__device__ __forceinline__ uint32_t mix32(uint32_t x) {  // lowbias32 integer hash
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// Shared memory of the gradient kernel: the weights once per block, then each warp's
// activations, transposed (row = unit, column = sample of the tile).
struct GradWeights {
  float w1t[kMlpIn][32];  // w1t[i][o] = w1[o][i]
  float w2t[32][36];      // w2t[k][o] = w2[o][k] (forward; rows padded against bank conflicts in the transposition)
  float w2[32][32];       // w2[o][k] (backward)
  float b1[32], b2[32], w3[32];
  float shift[kMlpIn], scale[kMlpIn];
  float b3, out_scale;
  float pad[2];
};
struct GradTile {
  float a[32][kLd];      // relu(z1), later the layer-1 deltas
  float d[32][kLd];      // layer-2 deltas
  float x[kMlpIn][kLd];  // normalised features
};
static_assert(sizeof(GradWeights) % 16 == 0 && sizeof(GradTile) % 16 == 0, "16-byte aligned rows");
static_assert(sizeof(GradTile) >= (kTrainable + 1) * sizeof(float), "a warp's gradient fits its tile");
constexpr size_t grad_smem(int warps) { return sizeof(GradWeights) + (size_t)warps * sizeof(GradTile); }

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}

// acc[j][u] += sum over the n rows k of in[k][sample j] * w[k][output u], for the lane's four
// samples (columns 4 sg ..) and eight outputs (8 og ..), two outputs per packed FMA (each
// rounded as the scalar one).
template <int kPitch>
__device__ __forceinline__ void tile_product(float (&acc)[4][8], const float (*in)[kLd], const float (*w)[kPitch], int n,
                                             int sg, int og) {
  float2 p[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int u = 0; u < 4; ++u) p[j][u] = make_float2(acc[j][2 * u], acc[j][2 * u + 1]);
#pragma unroll 2
  for (int k = 0; k < n; ++k) {
    const float4 sv4 = ld4(&in[k][4 * sg]);
    const float4 w0 = ld4(&w[k][8 * og]), w1 = ld4(&w[k][8 * og + 4]);
    const float sv[4] = {sv4.x, sv4.y, sv4.z, sv4.w};
    const float2 wv[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y), make_float2(w1.z, w1.w)};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int u = 0; u < 4; ++u) p[j][u] = __ffma2_rn(wv[u], make_float2(sv[j], sv[j]), p[j][u]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      acc[j][2 * u] = p[j][u].x;
      acc[j][2 * u + 1] = p[j][u].y;
    }
}
// Output u of the lane's tile for its four samples, as row `row` of a transposed buffer.
__device__ __forceinline__ void store_row(float (*out)[kLd], int row, const float (&acc)[4][8], int u, int sg) {
  st4(&out[row][4 * sg], acc[0][u], acc[1][u], acc[2][u], acc[3][u]);
}
// Sum of v[u] over the eight lanes sg = 0..7 that share og; lane sg gets entry u = sg.
__device__ __forceinline__ float sum_scatter(const float (&v)[8], int sg) {
  float a[4], b[2];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const bool up = sg & 4;
    a[u] = (up ? v[4 + u] : v[u]) + __shfl_xor_sync(0xffffffffu, up ? v[u] : v[4 + u], 4);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const bool up = sg & 2;
    b[u] = (up ? a[2 + u] : a[u]) + __shfl_xor_sync(0xffffffffu, up ? a[u] : a[2 + u], 2);
  }
  const bool up = sg & 1;
  return (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 1);
}

// Partial gradients of `count` samples of a batch of `total`: sample i is row first + i, or when
// `random` the row of [0, n) that the hash of first + i gives.  partial[block][0..kTrainable) gets
// the block's gradient sums, partial[block][kTrainable] its loss sum.  Tile t of 32
// samples belongs to block t % gridDim.x, warp t / gridDim.x (cyclically).
//
// What bounds it: instruction issue and latency at 3.5 warps per scheduler, beside the two launches
// of a step.  Each lane holds a 4 x 8 tile of
// the three passes (32 FMAs, two per instruction, from three 16-byte loads) and 8 x 4 of the
// 32 x 32 weight gradient (128 FMAs from twelve); the weight-gradient accumulators are kept
// over all of a warp's tiles, one FP32 chain each, of at most kMaxTilesPerWarp tiles.  One training step of 65,536 samples: 60.3 us with one
// thread per sample (every weight a broadcast load of its own, the weight gradients at two
// loads per FMA) and three launches; 25.5 us now.  With scalar FMAs 27.7 us; with 64-sample
// tiles (8 x 8 per lane, 7 warps per SM) 27.4 us without leaving room for the reduction's blocks.
__global__ void __launch_bounds__(32 * kMaxGradWarps, 1)
    grad_kernel(const float* params, const float* __restrict__ X, const float* __restrict__ T, long long n, long long first,
                long long count, long long total, int random, uint32_t seed, float* partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GradWeights& W = *reinterpret_cast<GradWeights*>(smem_raw);
  GradTile* tiles = reinterpret_cast<GradTile*>(smem_raw + sizeof(GradWeights));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int sg = lane & 7, og = lane >> 3;
  GradTile& s = tiles[warp];
  const int c0 = 4 * sg + og;  // this lane gathers sample c0 of a tile and evaluates its loss

  // the samples do not depend on the kernel ahead (which may still be updating the
  // parameters): fetch the first tile's before waiting for it.  Safe, also through read-only
  // loads, because both functions that add samples wait for the stream before they return.
  float2 raw[kMlpIn / 2] = {};
  float target = 0.f;
  bool valid = false;
  auto gather = [&](long long tile) {
    const long long i = tile * kTile + c0;
    valid = i < count;
    long long row = 0;
    if (valid) {
      row = first + i;
      if (random) {
        const uint32_t v = mix32(seed ^ mix32((uint32_t)row * 2654435761u + (uint32_t)(row >> 32)));
        row = n <= 0xffffffffll ? (long long)(v % (uint32_t)n) : (long long)v;
      }
    }
#pragma unroll
    for (int k = 0; k < kMlpIn / 2; ++k) raw[k] = reinterpret_cast<const float2*>(X + row * kMlpIn)[k];
    target = T[row];
  };
  long long tile = blockIdx.x + (long long)gridDim.x * warp;
  if (tile * kTile < count) gather(tile);

  grid_wait();
  grid_release();
  for (int base = threadIdx.x; base < kParams; base += 4 * blockDim.x) {  // one round at 14 warps
    float v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = base + c * blockDim.x;
      v[c] = i < kParams ? __ldcg(params + i) : 0.f;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = base + c * blockDim.x;
      if (i < kB1) W.w1t[i % kMlpIn][i / kMlpIn] = v[c];
      else if (i < kW2) W.b1[i - kB1] = v[c];
      else if (i < kB2) {
        W.w2[(i - kW2) >> 5][(i - kW2) & 31] = v[c];
        W.w2t[(i - kW2) & 31][(i - kW2) >> 5] = v[c];
      } else if (i < kW3) W.b2[i - kB2] = v[c];
      else if (i < kB3) W.w3[i - kW3] = v[c];
      else if (i < kShift) W.b3 = v[c];
      else if (i < kScale) W.shift[i - kShift] = v[c];
      else if (i < kOutScale) W.scale[i - kScale] = v[c];
      else if (i < kParams) W.out_scale = v[c];
    }
  }
  __syncthreads();

  const float inv_count = 1.f / (float)total;
  // gradient accumulators over the warp's tiles.  g2: rows o = og + 4 j, columns k = sg + 8 m;
  // g1: rows k = sg + 8 m, inputs 5 ig + i, half of the samples; b1, b2, w3: entry 8 og + sg
  const int ig = og & 1, half = og >> 1;
  float g2[8][4], g1[4][5], gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f, loss = 0.f;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
#pragma unroll
    for (int j = 0; j < 8; ++j) g2[j][m] = 0.f;
#pragma unroll
    for (int i = 0; i < 5; ++i) g1[m][i] = 0.f;
  }

  for (; tile * kTile < count; tile += (long long)gridDim.x * warps) {
    const bool ok = valid;
    const float t = target / W.out_scale;
#pragma unroll
    for (int k = 0; k < kMlpIn; ++k) {
      const float v = (k & 1) ? raw[k / 2].y : raw[k / 2].x;
      s.x[k][c0] = ok ? (v - W.shift[k]) * W.scale[k] : 0.f;
    }
    __syncwarp();
    float acc[4][8], sum[8];
    // ---- layer 1 ----
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][u] = W.b1[8 * og + u];
    tile_product(acc, s.x, W.w1t, kMlpIn, sg, og);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][u] = fmaxf(acc[j][u], 0.f);
      store_row(s.a, 8 * og + u, acc, u, sg);
    }
    __syncwarp();
    // ---- layer 2 and the output: z summed over the lane's outputs, then over the four lanes
    // that share its samples ----
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][u] = W.b2[8 * og + u];
    tile_product(acc, s.a, W.w2t, 32, sg, og);
    float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float w3 = W.w3[8 * og + u];
#pragma unroll
      for (int j = 0; j < 4; ++j) z[j] = fmaf(w3, fmaxf(acc[j][u], 0.f), z[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      z[j] += __shfl_xor_sync(0xffffffffu, z[j], 8);
      z[j] += __shfl_xor_sync(0xffffffffu, z[j], 16);
    }
    // each lane evaluates the loss of the sample it gathered; the four deltas come by shuffles
    const float zz = (og == 0 ? z[0] : og == 1 ? z[1] : og == 2 ? z[2] : z[3]) + W.b3;
    const float y = zz > 20.f ? zz : log1pf(expf(zz));
    const float r = ok ? y - t : 0.f;
    loss += r * r;
    const float dz_own = 2.f * r * inv_count / (1.f + expf(-fminf(zz, 50.f)));
    gb3 += dz_own;
    float dz[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) dz[j] = __shfl_sync(0xffffffffu, dz_own, sg + 8 * j);
    // ---- layer-2 deltas, and the sums over samples that need only them ----
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      sum[u] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[u] = fmaf(dz[j], fmaxf(acc[j][u], 0.f), sum[u]);
    }
    gw3 += sum_scatter(sum, sg);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float w3 = W.w3[8 * og + u];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][u] = acc[j][u] > 0.f ? dz[j] * w3 : 0.f;
      sum[u] = (acc[0][u] + acc[1][u]) + (acc[2][u] + acc[3][u]);
      store_row(s.d, 8 * og + u, acc, u, sg);
    }
    gb2 += sum_scatter(sum, sg);
    __syncwarp();
    // ---- weight gradient of layer 2: d (32 x samples) times a^T ----
#pragma unroll 1
    for (int c = 0; c < kTile; c += 4) {
      float4 av[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) av[m] = ld4(&s.a[sg + 8 * m][c]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 dv = ld4(&s.d[og + 4 * j][c]);
#pragma unroll
        for (int m = 0; m < 4; ++m)
          g2[j][m] = fmaf(dv.w, av[m].w, fmaf(dv.z, av[m].z, fmaf(dv.y, av[m].y, fmaf(dv.x, av[m].x, g2[j][m]))));
      }
    }
    // ---- layer-1 deltas ----
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][u] = 0.f;
    tile_product(acc, s.d, W.w2, 32, sg, og);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float4 a4 = ld4(&s.a[8 * og + u][4 * sg]);
      const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][u] = av[j] > 0.f ? acc[j][u] : 0.f;
      sum[u] = (acc[0][u] + acc[1][u]) + (acc[2][u] + acc[3][u]);
    }
    gb1 += sum_scatter(sum, sg);
    __syncwarp();  // every lane has read the activations that the deltas replace
#pragma unroll
    for (int u = 0; u < 8; ++u) store_row(s.a, 8 * og + u, acc, u, sg);
    __syncwarp();
    // the next tile's samples arrive during the last product
    const long long next = tile + (long long)gridDim.x * warps;
    if (next * kTile < count) gather(next);
    // ---- weight gradient of layer 1: d1 (32 x samples) times x^T ----
#pragma unroll 1
    for (int c = kTile / 2 * half; c < kTile / 2 * (half + 1); c += 4) {
      float4 dv[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) dv[m] = ld4(&s.a[sg + 8 * m][c]);
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const float4 xv = ld4(&s.x[5 * ig + i][c]);
#pragma unroll
        for (int m = 0; m < 4; ++m)
          g1[m][i] = fmaf(dv[m].w, xv.w, fmaf(dv[m].z, xv.z, fmaf(dv[m].y, xv.y, fmaf(dv[m].x, xv.x, g1[m][i]))));
      }
    }
    __syncwarp();  // the tile's buffers are free for the next one
  }

  // ---- the warp's sums, laid out like the parameters, into its own tile buffer ----
  float* mine = reinterpret_cast<float*>(&s);
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int m = 0; m < 4; ++m) mine[kW2 + (og + 4 * j) * 32 + sg + 8 * m] = g2[j][m];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float v = g1[m][i] + __shfl_xor_sync(0xffffffffu, g1[m][i], 16);
      if (half == 0) mine[kW1 + (sg + 8 * m) * kMlpIn + 5 * ig + i] = v;
    }
  mine[kB1 + 8 * og + sg] = gb1;
  mine[kB2 + 8 * og + sg] = gb2;
  mine[kW3 + 8 * og + sg] = gw3;
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    gb3 += __shfl_xor_sync(0xffffffffu, gb3, d);
    loss += __shfl_xor_sync(0xffffffffu, loss, d);
  }
  if (lane == 0) {
    mine[kB3] = gb3;
    mine[kTrainable] = loss;
  }
  __syncthreads();
  float* out = partial + (size_t)blockIdx.x * (kTrainable + 1);
  for (int e = threadIdx.x; e <= kTrainable; e += blockDim.x) {
    float v = 0.f;
    for (int w = 0; w < warps; ++w) v += reinterpret_cast<const float*>(&tiles[w])[e];
    out[e] = v;
  }
}

// grad[e] = sum over blocks of partial[block][e] in FP64, grad[kTrainable] the mean loss over
// `count`; with kAdam also the Adam update of the parameter.  Of a batch in pieces (not kWhole),
// every piece adds its sums to those of the pieces before it, and the last does the rest.  Eight entries (one 32-byte sector of a block's
// row) per block and 16 groups of threads that take every 16th row each, then the 16 sums in
// order.  One thread per entry summing all rows kept six blocks busy with a serial chain of
// loads (16.3 us at 296 rows, Adam a launch of its own at 4.2 us).  128 threads of at most 32
// registers fit beside a block of grad_kernel, so each of the two kernels is resident when
// the one ahead of it ends.
struct AdamParams {
  float* params;
  float* m;
  float* v;
  float lr, beta1, beta2, eps;
  int step;
};
struct PieceOf {
  bool first, last;
};
constexpr int kReduceEntries = 8, kReduceGroups = 16;
template <bool kAdam, bool kWhole>
__global__ void __launch_bounds__(kReduceEntries * kReduceGroups, 16)
    reduce_kernel(const float* partial, int blocks, long long count, PieceOf piece, double* grad, AdamParams ad) {
  __shared__ double part[kReduceGroups][kReduceEntries];
  const int entry = threadIdx.x % kReduceEntries, group = threadIdx.x / kReduceEntries;
  const int e = blockIdx.x * kReduceEntries + entry;
  grid_wait();
  grid_release();
  constexpr int kRows = (kGradBlocks + kReduceGroups - 1) / kReduceGroups;
  float v[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const int b = group + r * kReduceGroups;
    v[r] = e <= kTrainable && b < blocks ? __ldcg(partial + (size_t)b * (kTrainable + 1) + e) : 0.f;
  }
  double s = 0.0;
#pragma unroll
  for (int r = 0; r < kRows; ++r) s += (double)v[r];
  part[group][entry] = s;
  __syncthreads();
  if (group != 0 || e > kTrainable) return;
  s = 0.0;
#pragma unroll
  for (int w = 0; w < kReduceGroups; ++w) s += part[w][entry];
  if (!kWhole && !piece.first) s += grad[e];
  grad[e] = (kWhole || piece.last) && e == kTrainable ? s / (double)count : s;
  if (!kAdam || !(kWhole || piece.last) || e >= kTrainable) return;
  const float g = (float)s;
  const float mm = ad.beta1 * ad.m[e] + (1.f - ad.beta1) * g;
  const float vv = ad.beta2 * ad.v[e] + (1.f - ad.beta2) * g * g;
  ad.m[e] = mm;
  ad.v[e] = vv;
  const float mh = mm / (1.f - powf(ad.beta1, (float)ad.step));
  const float vh = vv / (1.f - powf(ad.beta2, (float)ad.step));
  ad.params[e] -= ad.lr * mh / (sqrtf(vh) + ad.eps);
}

// ---- samples from a fine periodic box ----
constexpr int kCoarseRecord = 19;  // 10 features, 3 filtered velocity, 6 subfilter stress

template <typename S>
__global__ void filter_kernel(GridView<S> fine, int fnx, int fny, int M, float* __restrict__ rec) {
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (long long)M * M * M) return;
  const int I = (int)(id % M), J = (int)((id / M) % M), K = (int)(id / ((long long)M * M));
  float f[27];
#pragma unroll
  for (int q = 0; q < 27; ++q) f[q] = 0.f;
  float uu[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int c = 0; c < 8; ++c) {
    const int i = 2 * I + (c & 1), j = 2 * J + ((c >> 1) & 1), k = 2 * K + (c >> 2);
    const uint32_t cell = ((uint32_t)k * fny + j) * fnx + i;
    float fc[27];
    load_cell<S>(fine, cell, fc);
    float rho = 0.f, jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll
    for (int q = 0; q < 27; ++q) {
      f[q] += fc[q];
      rho += fc[q];
      jx += cx(q) * fc[q];
      jy += cy(q) * fc[q];
      jz += cz(q) * fc[q];
    }
    const float ux = jx / rho, uy = jy / rho, uz = jz / rho;
    uu[0] += ux * ux;
    uu[1] += uy * uy;
    uu[2] += uz * uz;
    uu[3] += ux * uy;
    uu[4] += ux * uz;
    uu[5] += uy * uz;
  }
#pragma unroll
  for (int q = 0; q < 27; ++q) f[q] *= 0.125f;
  rescale(f, false);
  float Km[3][3][3];
  float rho, ux, uy, uz, inv_rho;
  central_moments(f, Km, rho, ux, uy, uz, inv_rho);
  float x[kMlpIn];
  mlp_features(Km[2][0][0], Km[0][2][0], Km[0][0][2], Km[1][1][0], Km[1][0][1], Km[0][1][1], rho, inv_rho, 1.f, x);
  float* r = rec + id * kCoarseRecord;
#pragma unroll
  for (int k = 0; k < kMlpIn; ++k) r[k] = x[k];
  r[10] = ux;
  r[11] = uy;
  r[12] = uz;
  r[13] = uu[0] * 0.125f - ux * ux;
  r[14] = uu[1] * 0.125f - uy * uy;
  r[15] = uu[2] * 0.125f - uz * uz;
  r[16] = uu[3] * 0.125f - ux * uy;
  r[17] = uu[4] * 0.125f - ux * uz;
  r[18] = uu[5] * 0.125f - uy * uz;
}

// Targets from the records (strain rate of the filtered velocity, periodic central
// differences) and the selected samples appended at X/T + `at`: cell `id` is selected when
// id % stride == phase.
__global__ void target_kernel(const float* __restrict__ rec, int M, int stride, int phase, float* __restrict__ X,
                              float* __restrict__ T, long long at) {
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (long long)M * M * M || id % stride != phase) return;
  const int I = (int)(id % M), J = (int)((id / M) % M), K = (int)(id / ((long long)M * M));
  auto u = [&](int i, int j, int k, int comp) {
    i = (i + M) % M;
    j = (j + M) % M;
    k = (k + M) % M;
    return rec[(((long long)k * M + j) * M + i) * kCoarseRecord + 10 + comp];
  };
  float g[3][3];  // g[a][b] = d u_b / d x_a
  for (int b = 0; b < 3; ++b) {
    g[0][b] = 0.5f * (u(I + 1, J, K, b) - u(I - 1, J, K, b));
    g[1][b] = 0.5f * (u(I, J + 1, K, b) - u(I, J - 1, K, b));
    g[2][b] = 0.5f * (u(I, J, K + 1, b) - u(I, J, K - 1, b));
  }
  float Sm[3][3];
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b) Sm[a][b] = 0.5f * (g[a][b] + g[b][a]);
  const float* r = rec + id * kCoarseRecord;
  const float tr = (r[13] + r[14] + r[15]) * (1.f / 3.f);
  const float tau[3][3] = {{r[13] - tr, r[16], r[17]}, {r[16], r[14] - tr, r[18]}, {r[17], r[18], r[15] - tr}};
  float ts = 0.f, ss = 0.f;
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b) {
      ts += tau[a][b] * Sm[a][b];
      ss += Sm[a][b] * Sm[a][b];
    }
  const float nu_t = fmaxf(0.f, -ts / (2.f * ss + 1e-30f));
  const long long slot = at + id / stride;
#pragma unroll
  for (int k = 0; k < kMlpIn; ++k) X[slot * kMlpIn + k] = r[k];
  T[slot] = nu_t;
}

void to_flat(const psl_sgs_mlp& m, float* p) {
  std::memcpy(p + kW1, m.w1, sizeof(m.w1));
  std::memcpy(p + kB1, m.b1, sizeof(m.b1));
  std::memcpy(p + kW2, m.w2, sizeof(m.w2));
  std::memcpy(p + kB2, m.b2, sizeof(m.b2));
  std::memcpy(p + kW3, m.w3, sizeof(m.w3));
  p[kB3] = m.b3;
  std::memcpy(p + kShift, m.in_shift, sizeof(m.in_shift));
  std::memcpy(p + kScale, m.in_scale, sizeof(m.in_scale));
  p[kOutScale] = m.out_scale;
}

void from_flat(const float* p, psl_sgs_mlp& m) {
  std::memcpy(m.w1, p + kW1, sizeof(m.w1));
  std::memcpy(m.b1, p + kB1, sizeof(m.b1));
  std::memcpy(m.w2, p + kW2, sizeof(m.w2));
  std::memcpy(m.b2, p + kB2, sizeof(m.b2));
  std::memcpy(m.w3, p + kW3, sizeof(m.w3));
  m.b3 = p[kB3];
  std::memcpy(m.in_shift, p + kShift, sizeof(m.in_shift));
  std::memcpy(m.in_scale, p + kScale, sizeof(m.in_scale));
  m.out_scale = p[kOutScale];
}

}  // namespace

struct psl_sgs_trainer {
  int device = 0;
  cudaStream_t stream = nullptr;
  long long capacity = 0, count = 0;
  float* X = nullptr;  // [capacity][10] raw features
  float* T = nullptr;  // [capacity] targets
  float* params = nullptr;  // kParams
  float* m = nullptr;       // Adam moments (kTrainable each)
  float* v = nullptr;
  int step = 0;
  float* partial = nullptr;  // [kGradBlocks][kTrainable + 1]
  double* grad = nullptr;    // kTrainable + 1
};

namespace {

// One warp per 32-sample tile while that many warps fit (14 per SM), so that a batch of 65,536
// samples is one tile per warp on 148 x 14 warps and a small batch spreads over the SMs; a batch of
// more than kPieceSamples in pieces of that size.
int run_gradient(psl_sgs_trainer* t, long long first, long long count, int random, uint32_t seed, const AdamParams* adam) {
  const unsigned int nb = (kTrainable + kReduceEntries) / kReduceEntries, threads = kReduceEntries * kReduceGroups;
  const bool whole = count <= kPieceSamples;
  const auto reduce = adam ? (whole ? reduce_kernel<true, true> : reduce_kernel<true, false>)
                           : (whole ? reduce_kernel<false, true> : reduce_kernel<false, false>);
  for (long long at = 0; at < count; at += kPieceSamples) {
    const long long samples = std::min(count - at, kPieceSamples), tiles = (samples + kTile - 1) / kTile;
    const int blocks = (int)std::min<long long>(kGradBlocks, tiles);
    const int warps = (int)std::min<long long>(kMaxGradWarps, (tiles + blocks - 1) / blocks);
    TRAIN_CUDA(launch_dependent(true, grad_kernel, dim3(blocks), 32 * warps, grad_smem(warps), t->stream,
                                (const float*)t->params, (const float*)t->X, (const float*)t->T, t->count, first + at, samples, count,
                                random, seed, t->partial));
    const PieceOf piece{at == 0, at + samples == count};
    TRAIN_CUDA(launch_dependent(true, reduce, dim3(nb), threads, 0, t->stream, (const float*)t->partial, blocks, count, piece,
                                t->grad, adam ? *adam : AdamParams{}));
  }
  return PSL_OK;
}

}  // namespace

int psl_sgs_trainer_create(long long capacity, psl_sgs_trainer** out) {
  if (!out || capacity <= 0) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_create: bad argument");
  *out = nullptr;
  int ndev = 0;
  TRAIN_CUDA(cudaGetDeviceCount(&ndev));
  if (ndev <= 0) return fail(PSL_ERR_CUDA, "psl_sgs_trainer_create: no CUDA device");
  psl_sgs_trainer* t = new psl_sgs_trainer();
  cudaGetDevice(&t->device);
  t->capacity = capacity;
  cudaError_t e = cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&t->X, (size_t)capacity * kMlpIn * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&t->T, (size_t)capacity * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&t->params, kParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&t->m, kTrainable * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&t->v, kTrainable * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&t->partial, (size_t)kGradBlocks * (kTrainable + 1) * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&t->grad, (kTrainable + 1) * sizeof(double));
  if (e == cudaSuccess) e = cudaMemset(t->params, 0, kParams * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(t->m, 0, kTrainable * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(t->v, 0, kTrainable * sizeof(float));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grad_smem(kMaxGradWarps));
  if (e != cudaSuccess) {
    const std::string msg = std::string("psl_sgs_trainer_create: ") + cudaGetErrorString(e);
    cudaGetLastError();
    psl_sgs_trainer_destroy(t);
    return fail(e == cudaErrorMemoryAllocation ? PSL_ERR_NOMEM : PSL_ERR_CUDA, msg);
  }
  *out = t;
  return PSL_OK;
}

int psl_sgs_trainer_destroy(psl_sgs_trainer* t) {
  if (!t) return PSL_OK;
  DeviceGuard dg(t->device);
  if (t->stream) cudaStreamSynchronize(t->stream);
  for (void* p : {(void*)t->X, (void*)t->T, (void*)t->params, (void*)t->m, (void*)t->v, (void*)t->partial, (void*)t->grad})
    if (p) cudaFree(p);
  if (t->stream) cudaStreamDestroy(t->stream);
  delete t;
  return PSL_OK;
}

int psl_sgs_trainer_clear(psl_sgs_trainer* t) {
  if (!t) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_clear: null trainer");
  t->count = 0;
  return PSL_OK;
}

int psl_sgs_trainer_count(const psl_sgs_trainer* t, long long* count) {
  if (!t || !count) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_count: null argument");
  *count = t->count;
  return PSL_OK;
}

int psl_sgs_trainer_add_samples(psl_sgs_trainer* t, const float* features, const float* targets, long long n) {
  if (!t || !features || !targets || n < 0) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_add_samples: bad argument");
  if (t->count + n > t->capacity) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_add_samples: capacity exceeded");
  DeviceGuard dg(t->device);
  TRAIN_CUDA(cudaMemcpyAsync(t->X + t->count * kMlpIn, features, (size_t)n * kMlpIn * sizeof(float),
                             cudaMemcpyHostToDevice, t->stream));
  TRAIN_CUDA(cudaMemcpyAsync(t->T + t->count, targets, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, t->stream));
  TRAIN_CUDA(cudaStreamSynchronize(t->stream));  // required: grad_kernel reads samples before its grid_wait
  t->count += n;
  return PSL_OK;
}

int psl_sgs_trainer_get_samples(psl_sgs_trainer* t, long long first, long long n, float* features, float* targets) {
  if (!t || first < 0 || n < 0 || first + n > t->count) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_get_samples: bad range");
  DeviceGuard dg(t->device);
  if (features)
    TRAIN_CUDA(cudaMemcpyAsync(features, t->X + first * kMlpIn, (size_t)n * kMlpIn * sizeof(float),
                               cudaMemcpyDeviceToHost, t->stream));
  if (targets)
    TRAIN_CUDA(cudaMemcpyAsync(targets, t->T + first, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost, t->stream));
  TRAIN_CUDA(cudaStreamSynchronize(t->stream));
  return PSL_OK;
}

int psl_sgs_trainer_add_filtered(psl_sgs_trainer* t, psl_grid* fine, int M, int stride, unsigned int phase) {
  if (!t || !fine || M < 2 || stride < 1) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_add_filtered: bad argument");
  const psl_info& I = fine->info;
  if (I.cell_count_x != 2 * M + 1 || I.cell_count_y != 2 * M + 1 || I.cell_count_z != 2 * M)
    return fail(PSL_ERR_INVALID, "psl_sgs_trainer_add_filtered: fine grid must be (2M+1) x (2M+1) x 2M (periodic box)");
  if (fine->storage == kStoreF64) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_add_filtered: FP64 storage");
  const long long cells = (long long)M * M * M;
  const long long selected = (cells - (long long)(phase % stride) + stride - 1) / stride;
  if (t->count + selected > t->capacity) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_add_filtered: capacity exceeded");
  DeviceGuard dg(t->device);
  float* rec = nullptr;
  TRAIN_CUDA(cudaMalloc(&rec, (size_t)cells * kCoarseRecord * sizeof(float)));
  TRAIN_CUDA(cudaStreamSynchronize(fine->stream));
  const unsigned int nb = (unsigned int)((cells + 255) / 256);
  auto go = [&](auto s) {
    using S = decltype(s);
    GridView<S> v;
    typename S::type* base = static_cast<typename S::type*>(fine->f);
    for (int q = 0; q < 27; ++q) {
      v.fq[q] = base + (size_t)q * fine->f_stride;
      v.shift[q] = fine->shift[q];
    }
    v.n = fine->n;
    filter_kernel<S><<<nb, 256, 0, t->stream>>>(v, I.cell_count_x, I.cell_count_y, M, rec);
  };
  switch (fine->storage) {
    case kStoreF32: go(StoreF32{}); break;
    case kStoreF16: go(StoreF16{}); break;
    default: go(StoreBF16{}); break;
  }
  target_kernel<<<nb, 256, 0, t->stream>>>(rec, M, stride, (int)(phase % stride), t->X, t->T, t->count);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);  // required: grad_kernel reads samples before its grid_wait
  cudaFree(rec);
  if (e != cudaSuccess) return fail(PSL_ERR_CUDA, std::string("psl_sgs_trainer_add_filtered: ") + cudaGetErrorString(e));
  t->count += selected;
  return PSL_OK;
}

int psl_sgs_trainer_set_params(psl_sgs_trainer* t, const psl_sgs_mlp* mlp) {
  if (!t || !mlp) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_set_params: null argument");
  DeviceGuard dg(t->device);
  std::vector<float> p(kParams);
  to_flat(*mlp, p.data());
  TRAIN_CUDA(cudaMemcpyAsync(t->params, p.data(), kParams * sizeof(float), cudaMemcpyHostToDevice, t->stream));
  TRAIN_CUDA(cudaMemsetAsync(t->m, 0, kTrainable * sizeof(float), t->stream));
  TRAIN_CUDA(cudaMemsetAsync(t->v, 0, kTrainable * sizeof(float), t->stream));
  TRAIN_CUDA(cudaStreamSynchronize(t->stream));
  t->step = 0;
  return PSL_OK;
}

int psl_sgs_trainer_get_params(psl_sgs_trainer* t, psl_sgs_mlp* mlp) {
  if (!t || !mlp) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_get_params: null argument");
  DeviceGuard dg(t->device);
  std::vector<float> p(kParams);
  TRAIN_CUDA(cudaMemcpyAsync(p.data(), t->params, kParams * sizeof(float), cudaMemcpyDeviceToHost, t->stream));
  TRAIN_CUDA(cudaStreamSynchronize(t->stream));
  from_flat(p.data(), *mlp);
  return PSL_OK;
}

int psl_sgs_trainer_gradient(psl_sgs_trainer* t, long long first, long long count, psl_sgs_mlp* grad, double* loss) {
  if (!t || first < 0 || count <= 0 || first + count > t->count)
    return fail(PSL_ERR_INVALID, "psl_sgs_trainer_gradient: bad range");
  DeviceGuard dg(t->device);
  int rc = run_gradient(t, first, count, 0, 0, nullptr);
  if (rc) return rc;
  std::vector<double> g(kTrainable + 1);
  TRAIN_CUDA(cudaMemcpyAsync(g.data(), t->grad, (kTrainable + 1) * sizeof(double), cudaMemcpyDeviceToHost, t->stream));
  TRAIN_CUDA(cudaStreamSynchronize(t->stream));
  if (grad) {
    std::vector<float> p(kParams, 0.f);
    for (int e = 0; e < kTrainable; ++e) p[e] = (float)g[e];
    from_flat(p.data(), *grad);
  }
  if (loss) *loss = g[kTrainable];
  return PSL_OK;
}

int psl_sgs_trainer_train(psl_sgs_trainer* t, int steps, int batch, float lr, unsigned int seed, double* last_loss) {
  if (!t || steps < 0 || batch <= 0 || t->count <= 0) return fail(PSL_ERR_INVALID, "psl_sgs_trainer_train: bad argument");
  DeviceGuard dg(t->device);
  for (int s = 0; s < steps; ++s) {
    ++t->step;
    const AdamParams adam{t->params, t->m, t->v, lr, 0.9f, 0.999f, 1e-8f, t->step};
    int rc = run_gradient(t, 0, batch, 1, seed * 0x9e3779b9u + (uint32_t)t->step, &adam);
    if (rc) return rc;
  }
  TRAIN_CUDA(cudaGetLastError());
  if (last_loss) {
    TRAIN_CUDA(cudaMemcpyAsync(last_loss, t->grad + kTrainable, sizeof(double), cudaMemcpyDeviceToHost, t->stream));
  }
  TRAIN_CUDA(cudaStreamSynchronize(t->stream));
  return PSL_OK;
}
