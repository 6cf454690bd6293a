// Learned path guiding: network initialisation and packing, tensor-core
// forward pass for given features, and the training step.
//
// Training is a hand-written FP32 pipeline over a batch of samples: the
// forward pass layer by layer (inputs of every layer kept), the mixture loss
// gradient per sample, the backward pass layer by layer, and weight gradients
// as per-chunk partial sums reduced in a fixed order, so a step's gradients do
// not depend on scheduling. Adam then updates the FP32 master weights, which
// are repacked as the BF16 tensor-core operand image for inference.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "dev_common.cuh"
#include "guide.h"
#include "guide_mlp.cuh"
#include "guide_tc.cuh"

namespace muon_gpu {

namespace {

using namespace guide;

constexpr int kThreads = 256;
// Weight gradients are partial sums of at most kMaxChunks chunks of samples
// (two blocks for each of 152 SMs; a constant, so that the order of the sums,
// and with it every bit of a trained network, follows from the batch alone),
// reduced in order afterwards. Fixed chunks
// of 512 samples left a batch of 65,536 with 128 blocks: a 64 x 64 layer 57 us,
// now 24, the first 123, now 86.
constexpr int kMaxChunks = 304;
inline int ChunkSamples(int batch) {
  const int c = (batch + kMaxChunks - 1) / kMaxChunks;
  return (std::max(c, 64) + 31) / 32 * 32;
}
inline int Chunks(int batch) { return (batch + ChunkSamples(batch) - 1) / ChunkSamples(batch); }

// ---- packing and initialisation ------------------------------------------------
// The inference image (guide_mlp.cuh): one thread per 16-byte chunk of a
// layer's operand (8 BF16 weights of one output along K) or per bias.
constexpr int kImgChunks = kImgBiasOffset / 16;

__global__ void PackKernel(const float *params, unsigned char *img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kImgChunks) {
    const int byte = 16 * i;
    int l = 0;
    while (l + 1 < kLayers && byte >= ImgOffset(l + 1)) ++l;
    const int K = In(l);
    const int local = byte - ImgOffset(l);
    const int rb = local / ((K / 8) * 128), rem = local % ((K / 8) * 128);
    const int kb = rem / 128, r = rb * 8 + (rem % 128) / 16;
    uint32_t w[4];
    for (int e = 0; e < 4; ++e) {
      const int k = 8 * kb + 2 * e;
      float lo = 0.0f, hi = 0.0f;
      if (r < Out(l)) {
        lo = params[MasterOffset(l) + k * Out(l) + r];
        hi = params[MasterOffset(l) + (k + 1) * Out(l) + r];
      }
      w[e] = PackBf16(lo, hi);
    }
    *reinterpret_cast<uint4 *>(img + byte) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  if (i < kBiasFloats) {
    const int l = i < 4 * kWidth ? i / kWidth : kLayers - 1;
    const int o = i - BiasOffset(l);
    reinterpret_cast<float *>(img + kImgBiasOffset)[i] = params[MasterOffset(l) + In(l) * Out(l) + o];
  }
}

// He-uniform weights U(-sqrt(6 / fan_in), sqrt(6 / fan_in)), zero biases.
__global__ void InitKernel(float *params, uint64_t seed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  int l = 0;
  while (l + 1 < kLayers && i >= MasterOffset(l + 1)) ++l;
  const int local = i - MasterOffset(l);
  if (local >= In(l) * Out(l)) {
    params[i] = 0.0f;
    return;
  }
  Rng r(seed, 0, 0);
  r.ctr = make_uint4(static_cast<uint32_t>(i), 0x6d6c70u, 0u, 0u);
  const float lim = sqrtf(6.0f / static_cast<float>(In(l)));
  params[i] = (2.0f * r.Next() - 1.0f) * lim;
}

// ---- tensor-core forward for given features ------------------------------------
// The inference kernel's network pass (guide_tc.cuh) over features read from
// memory: one CTA per SM, 128 rows per group.
__global__ void __launch_bounds__(kTcThreads, 1) ForwardKernel(const void *img, const float *features, int n,
                                                               float *out, int32_t *status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if (static_cast<int>(blockIdx.x) * kTcThreads >= n) return;  // the whole CTA
  TcGroup grp;
  bool ok = TcBegin(smem, img, &grp);
  const int group = threadIdx.x / kTcRows;
  for (int base = (blockIdx.x * 2 + group) * kTcRows; ok && base < n; base += gridDim.x * kTcThreads) {
    const int r = base + grp.row;
    float f[kFeatures];
#pragma unroll
    for (int d = 0; d < kFeatures; ++d) f[d] = r < n ? features[static_cast<int64_t>(r) * kFeatures + d] : 0.0f;
    float o[kOut];
    ok = TcForward(grp, f, o);
    if (ok && r < n)
#pragma unroll
      for (int c = 0; c < kOut; ++c) out[static_cast<int64_t>(r) * kOut + c] = o[c];
  }
  TcEnd(smem, grp, status);
}

// T consecutive floats of shared memory into registers, as 16- or 8-byte
// loads where T allows (p is aligned to T floats).
template <int T>
__device__ __forceinline__ void LoadRow(const float *p, float (&v)[T]) {
  if constexpr (T % 4 == 0) {
#pragma unroll
    for (int q = 0; q < T / 4; ++q) {
      const float4 f = reinterpret_cast<const float4 *>(p)[q];
      v[4 * q] = f.x, v[4 * q + 1] = f.y, v[4 * q + 2] = f.z, v[4 * q + 3] = f.w;
    }
  } else if constexpr (T % 2 == 0) {
#pragma unroll
    for (int q = 0; q < T / 2; ++q) {
      const float2 f = reinterpret_cast<const float2 *>(p)[q];
      v[2 * q] = f.x, v[2 * q + 1] = f.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < T; ++q) v[q] = p[q];
  }
}

// ---- sampling the mixture for given network outputs ------------------------------
__global__ void MixKernel(const float *raw, int n, float *mix) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) MakeMixture(raw + static_cast<int64_t>(i) * kOut, mix + static_cast<int64_t>(i) * kMixFloats);
}

__global__ void SampleKernel(const float *mix, int n, const float *u, float *dirs, float *pdf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float *mx = mix + static_cast<int64_t>(i) * kMixFloats;
  float wx, wy, wz;
  SampleMixture(mx, u[3 * i], u[3 * i + 1], u[3 * i + 2], &wx, &wy, &wz);
  dirs[3 * i] = wx, dirs[3 * i + 1] = wy, dirs[3 * i + 2] = wz;
  pdf[i] = MixturePdf(mx, wx, wy, wz);
}

// ---- training: layer products -----------------------------------------------------
// The forward and the data-gradient kernels multiply a tile of 128 samples by a
// 64 x 64 weight block with 128 threads, 8 x 8 outputs each, 32 inputs at a
// time. Both operands lie in shared memory with the summed index outermost, so
// that a thread's 16 operands of one step are four 16-byte loads for 64
// multiply-adds (4 x 4 outputs took five loads for 16). The 128-sample rows are
// stored with bits 2..4 of the column flipped by bits 2..4 of the row: writes
// of a transposed tile then hit all banks, and groups of four stay together.
// Every output sums its inputs in order, as one chain of multiply-adds. Bound
// by the FP32 units and, at 512 tiles, by the wait for each piece: 65,536
// samples x 64 x 64 forward 27 -> 20 us, backward 38 -> 22 (0.54 GFLOP, 27
// TFLOP/s).
constexpr int kTile = 128, kTileThreads = 128, kStep = 32;

__device__ __forceinline__ int Swizzle(int row) { return ((row >> 2) & 7) << 2; }

// acc[i][j] += sum over kStep rows r of xs[r][8 ty + i] * ws[r][8 tx + j].
__device__ __forceinline__ void TileProduct(const float (*xs)[kTile], const float (*ws)[64], int ty, int tx,
                                            bool ws_swizzled, float (&acc)[8][8]) {
#pragma unroll 8
  for (int r = 0; r < kStep; ++r) {
    const int sw = Swizzle(r);
    const float4 a0 = *reinterpret_cast<const float4 *>(&xs[r][(8 * ty) ^ sw]);
    const float4 a1 = *reinterpret_cast<const float4 *>(&xs[r][(8 * ty + 4) ^ sw]);
    const int wsw = ws_swizzled ? sw : 0;
    const float4 b0 = *reinterpret_cast<const float4 *>(&ws[r][(8 * tx) ^ wsw]);
    const float4 b1 = *reinterpret_cast<const float4 *>(&ws[r][(8 * tx + 4) ^ wsw]);
    const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  }
}

// xs[k][b] = x[b0 + b][k0 + k] for a 128 x 32 piece of a batch x 64 array.
__device__ __forceinline__ void LoadTransposed(const float *x, int b0, int k0, int batch, float (*xs)[kTile]) {
  const int c4 = threadIdx.x & 7, r0 = threadIdx.x >> 3;  // 8 vectors a row, 16 rows at a time
#pragma unroll
  for (int m = 0; m < kTile / 16; ++m) {
    const int row = r0 + 16 * m, b = b0 + row;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (b < batch) v = *reinterpret_cast<const float4 *>(x + static_cast<int64_t>(b) * kWidth + k0 + 4 * c4);
    const int col = row ^ (c4 << 2);
    xs[4 * c4][col] = v.x, xs[4 * c4 + 1][col] = v.y, xs[4 * c4 + 2][col] = v.z, xs[4 * c4 + 3][col] = v.w;
  }
}

// ---- training: forward ----------------------------------------------------------
// y[b][n] = act(sum_k x[b][k] w[k][n] + bias[n]), 64 outputs; with kBlob, x is
// the one-blob encoding of features (batch x 8), one feature per step.
template <bool kBlob, bool kRelu>
__global__ void __launch_bounds__(kTileThreads) FwdLayerKernel(const float *x, const float *w, const float *bias, int K,
                                                               float *y, int batch) {
  static_assert(kBins == kStep && kWidth == 64 && kOut == 64, "one feature a step, 64 outputs");
  __shared__ __align__(16) float xs[kStep][kTile];
  __shared__ __align__(16) float ws[kStep][64];
  const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
  const int b0 = blockIdx.x * kTile;
  float acc[8][8] = {};
  for (int k0 = 0; k0 < K; k0 += kStep) {
    if (kBlob) {
      const int b = b0 + tid;
      const bool on = b < batch;
      const float f = on ? x[static_cast<int64_t>(b) * kFeatures + k0 / kBins] : 0.0f;
#pragma unroll 8
      for (int k = 0; k < kBins; ++k) xs[k][tid ^ Swizzle(k)] = on ? Blob(f, k) : 0.0f;
    } else {
      LoadTransposed(x, b0, k0, batch, xs);
    }
#pragma unroll
    for (int i = tid; i < kStep * 16; i += kTileThreads)
      reinterpret_cast<float4 *>(&ws[0][0])[i] = reinterpret_cast<const float4 *>(w + k0 * 64)[i];
    __syncthreads();
    TileProduct(xs, ws, ty, tx, false, acc);
    __syncthreads();
  }
  float bb[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) bb[j] = bias[8 * tx + j];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int b = b0 + 8 * ty + i;
    if (b >= batch) continue;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = kRelu ? fmaxf(acc[i][j] + bb[j], 0.0f) : acc[i][j] + bb[j];
    float4 *o = reinterpret_cast<float4 *>(y + static_cast<int64_t>(b) * 64 + 8 * tx);
    o[0] = make_float4(v[0], v[1], v[2], v[3]), o[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// ---- training: loss ---------------------------------------------------------------
// Replaces z (raw outputs) by d(mean loss)/dz and writes per-block loss sums.
// Per sample: loss -weight log q(w) and its gradient with respect to the 64
// raw outputs (written over them), mean over the batch. q = (1 - eps)
// sum_i pi_i p_i + eps / (4 pi) with the lobes of guide_mlp.cuh; the
// gradient of log p_i follows oracle/guiding.py (loss_grad), through
// s = exp(b) (inside the clip range), the tangent projection pu = u - (u.mu) mu
// and mu = m / |m|.
// Eight lanes per sample, one per lobe: a lane reads and writes its lobe's 32
// bytes (a thread per sample read rows 256 bytes apart and walked the lobes in
// turn: 50 us for 65,536 samples, now 19).
__device__ __forceinline__ float LobeSum(float v) {
  for (int o = 1; o < kLobes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float LobeMax(float v) {
  for (int o = 1; o < kLobes; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__global__ void __launch_bounds__(kThreads) LossKernel(float *z, const float *dirs, const float *weights, int batch,
                                                       double *loss_out) {
  static_assert(kThreads == kLobes * kGuideLossSamples, "one loss sum per block");
  __shared__ double red[kGuideLossSamples];
  const int lobe = threadIdx.x & (kLobes - 1), sample = threadIdx.x / kLobes;
  const int b = blockIdx.x * kGuideLossSamples + sample;
  const bool on = b < batch;
  float r[kLobeOut] = {};
  float w[3] = {0.0f, 0.0f, 1.0f}, wt = 0.0f;
  float4 *row = reinterpret_cast<float4 *>(z + static_cast<int64_t>(b) * kOut + kLobeOut * lobe);
  if (on) {
    const float4 r0 = row[0], r1 = row[1];
    r[0] = r0.x, r[1] = r0.y, r[2] = r0.z, r[3] = r0.w, r[4] = r1.x, r[5] = r1.y, r[6] = r1.z, r[7] = r1.w;
    w[0] = dirs[3 * static_cast<int64_t>(b)], w[1] = dirs[3 * static_cast<int64_t>(b) + 1];
    w[2] = dirs[3 * static_cast<int64_t>(b) + 2];
    wt = weights[b];
  }
  const float amax = LobeMax(r[0]);
  const float lse = amax + logf(LobeSum(expf(r[0] - amax)));
  // log of the lobe's share of q (-inf where the lobe is zero)
  const float log_keep = logf(1.0f - kEpsUniform), t_uniform = logf(kEpsUniform * 0.25f / kPi);
  float t = -INFINITY;
  const float n2 = r[1] * r[1] + r[2] * r[2] + r[3] * r[3];
  const float nrm = sqrtf(n2);
  float mu[3] = {0.0f, 0.0f, 1.0f};
  if (n2 > 1e-24f) mu[0] = r[1] / nrm, mu[1] = r[2] / nrm, mu[2] = r[3] / nrm;
  const float c = mu[0] * w[0] + mu[1] * w[1] + mu[2] * w[2];
  const float s = expf(fminf(fmaxf(r[4], kBMin), kBMax));
  const float um = r[5] * mu[0] + r[6] * mu[1] + r[7] * mu[2];
  float pu[3], v[3], p2 = 0.0f, v2 = 0.0f, d = 0.0f, vw = 0.0f, pw = 0.0f;
  if (c > kCMin) {
    for (int k = 0; k < 3; ++k) {
      pu[k] = r[5 + k] - um * mu[k];
      v[k] = w[k] / c - mu[k];
      p2 += pu[k] * pu[k], v2 += v[k] * v[k], d += pu[k] * v[k];
      vw += v[k] * w[k], pw += pu[k] * w[k];
    }
    const float logp = 0.5f * logf(s) + 0.5f * logf(s + p2) - logf(2.0f * kPi) - 0.5f * (s * v2 + d * d) - 3.0f * logf(c);
    t = log_keep + (r[0] - lse) + logp;
  }
  const float tmax = fmaxf(t_uniform, LobeMax(t));
  const float logq = tmax + logf(expf(t_uniform - tmax) + LobeSum(expf(t - tmax)));
  const float resp = expf(t - logq);
  const float rsum = LobeSum(resp);
  if (on) {
    const float coef = -wt / static_cast<float>(batch);
    const float pi = expf(r[0] - lse);
    float g[kLobeOut] = {coef * (resp - pi * rsum), 0, 0, 0, 0, 0, 0, 0};
    if (resp > 0.0f && c > kCMin) {
      const float cr = coef * resp;
      const float sp2 = s + p2;
      if (r[4] > kBMin && r[4] < kBMax) g[4] = cr * (0.5f + 0.5f * s / sp2 - 0.5f * s * v2);
      for (int k = 0; k < 3; ++k) g[5 + k] = cr * (pu[k] / sp2 - d * v[k]);
      if (n2 > 1e-24f) {
        const float ic2 = 1.0f / (c * c);
        float gm[3], dot = 0.0f;
        for (int k = 0; k < 3; ++k) {
          gm[k] = -um * pu[k] / sp2 + s * (vw * w[k] * ic2 + v[k]) + d * (um * v[k] + pw * w[k] * ic2 + pu[k]) -
                  3.0f * w[k] / c;
          dot += gm[k] * mu[k];
        }
        for (int k = 0; k < 3; ++k) g[1 + k] = cr * (gm[k] - dot * mu[k]) / nrm;
      }
    }
    row[0] = make_float4(g[0], g[1], g[2], g[3]);
    row[1] = make_float4(g[4], g[5], g[6], g[7]);
  }
  if (lobe == 0) red[sample] = on ? -static_cast<double>(wt) * logq : 0.0;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int i = 0; i < kGuideLossSamples; ++i) sum += red[i];
    loss_out[blockIdx.x] = sum;
  }
}

// ---- training: backward -------------------------------------------------------------
// dx[b][k] = (sum_n dz[b][n] w[k][n]) * (h[b][k] > 0), 64 inputs and outputs.
__global__ void __launch_bounds__(kTileThreads) BwdDataKernel(const float *dz, const float *w, const float *h,
                                                              float *dx, int batch) {
  __shared__ __align__(16) float ds[kStep][kTile];
  __shared__ __align__(16) float wt[kStep][64];  // wt[n][k] = w[k][n], columns flipped as in ds
  const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
  const int b0 = blockIdx.x * kTile;
  float acc[8][8] = {};
  for (int n0 = 0; n0 < 64; n0 += kStep) {
    LoadTransposed(dz, b0, n0, batch, ds);
    const int c4 = tid & 7;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int k = (tid >> 3) + 16 * m;
      const float4 v = *reinterpret_cast<const float4 *>(w + k * 64 + n0 + 4 * c4);
      const int col = k ^ (c4 << 2);
      wt[4 * c4][col] = v.x, wt[4 * c4 + 1][col] = v.y, wt[4 * c4 + 2][col] = v.z, wt[4 * c4 + 3][col] = v.w;
    }
    __syncthreads();
    TileProduct(ds, wt, ty, tx, true, acc);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int b = b0 + 8 * ty + i;
    if (b >= batch) continue;
    const int64_t o = static_cast<int64_t>(b) * kWidth + 8 * tx;
    const float4 h0 = *reinterpret_cast<const float4 *>(h + o), h1 = *reinterpret_cast<const float4 *>(h + o + 4);
    *reinterpret_cast<float4 *>(dx + o) = make_float4(h0.x > 0.0f ? acc[i][0] : 0.0f, h0.y > 0.0f ? acc[i][1] : 0.0f,
                                                      h0.z > 0.0f ? acc[i][2] : 0.0f, h0.w > 0.0f ? acc[i][3] : 0.0f);
    *reinterpret_cast<float4 *>(dx + o + 4) =
        make_float4(h1.x > 0.0f ? acc[i][4] : 0.0f, h1.y > 0.0f ? acc[i][5] : 0.0f, h1.z > 0.0f ? acc[i][6] : 0.0f,
                    h1.w > 0.0f ? acc[i][7] : 0.0f);
  }
}

// Weight and bias gradients of a 64 x 64 layer over one chunk of samples:
// partial[k][n] = sum_b x[b][k] dz[b][n], then sum_b dz[b][n]. Four groups of 64
// threads take every fourth sample of the staged 32, 8 x 8 gradients a thread
// (four 16-byte loads for 64 multiply-adds), and their sums are added in order
// at the end; the next 32 samples load meanwhile.
constexpr int kSlices = kThreads / 64;
__global__ void __launch_bounds__(kThreads, 2) WgradSquareKernel(const float *x, const float *dz, int batch,
                                                                 int chunk, float *partial, int layer_off) {
  constexpr int kRows = 32, kVec = kRows * 64 / 4 / kThreads;  // rows staged, vectors a thread
  __shared__ __align__(16) float xs[kRows][64], ds[kRows][64];
  __shared__ float sums[64][65];
  const int tid = threadIdx.x, slice = tid >> 6, kg = (tid >> 3) & 7, ng = tid & 7;
  const int b0 = blockIdx.x * chunk, b1 = min(batch, b0 + chunk);
  float acc[8][8] = {}, bacc[8] = {};
  float4 px[kVec], pd[kVec];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int m = 0; m < kVec; ++m) {
      const int i = tid + m * kThreads, b = s0 + (i >> 4);
      px[m] = pd[m] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (b < b1) {
        px[m] = reinterpret_cast<const float4 *>(x + static_cast<int64_t>(b) * 64)[i & 15];
        pd[m] = reinterpret_cast<const float4 *>(dz + static_cast<int64_t>(b) * 64)[i & 15];
      }
    }
  };
  fetch(b0);
  for (int s0 = b0; s0 < b1; s0 += kRows) {
#pragma unroll
    for (int m = 0; m < kVec; ++m) {
      const int i = tid + m * kThreads;
      reinterpret_cast<float4 *>(&xs[0][0])[i] = px[m];
      reinterpret_cast<float4 *>(&ds[0][0])[i] = pd[m];
    }
    __syncthreads();
    if (s0 + kRows < b1) fetch(s0 + kRows);
#pragma unroll 4
    for (int r = slice; r < kRows; r += kSlices) {
      float a[8], d[8];
      LoadRow<8>(&xs[r][8 * kg], a);
      LoadRow<8>(&ds[r][8 * ng], d);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], d[j], acc[i][j]);
      if (kg == 0)
#pragma unroll
        for (int j = 0; j < 8; ++j) bacc[j] += d[j];
    }
    __syncthreads();
  }
  // rows 0..63: weights; the bias row through the last column
  float *p = partial + static_cast<int64_t>(blockIdx.x) * kParams + layer_off;
  for (int q = 0; q < kSlices; ++q) {
    if (slice == q) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float &o = sums[8 * kg + i][8 * ng + j];
          o = q == 0 ? acc[i][j] : o + acc[i][j];
        }
      if (kg == 0)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float &o = sums[8 * ng + j][64];
          o = q == 0 ? bacc[j] : o + bacc[j];
        }
    }
    __syncthreads();
  }
  for (int i = tid; i < 64 * 64; i += kThreads) p[i] = sums[i >> 6][i & 63];
  if (tid < 64) p[64 * 64 + tid] = sums[tid][64];
}

// The same for the first layer, whose inputs are the one-blob encoding: each
// thread owns an 8 x 8 tile of the 256 x 64 gradient; 32 samples at a time are
// staged in shared memory (rows of inputs and of outputs, read back as vectors).
__global__ void __launch_bounds__(kThreads) WgradBlobKernel(const float *features, const float *dz, int batch,
                                                            int chunk, float *partial, int layer_off) {
  constexpr int K = kIn, N = kWidth, T = 8;
  static_assert((K / T) * (N / T) == kThreads, "thread tiling");
  __shared__ __align__(16) float xs[32][K];
  __shared__ __align__(16) float ds[32][N];
  __shared__ float fs[32][kFeatures];  // the slab's features
  const int tid = threadIdx.x;
  const int kg = tid / (N / T), ng = tid % (N / T);
  const int b0 = blockIdx.x * chunk;
  float acc[T][T] = {};
  float bacc = 0.0f;
  for (int s0 = b0; s0 < b0 + chunk && s0 < batch; s0 += 32) {
    for (int i = tid; i < 32 * kFeatures; i += kThreads) {
      const int r = i / kFeatures, b = s0 + r;
      fs[r][i % kFeatures] = b < batch ? features[static_cast<int64_t>(b) * kFeatures + i % kFeatures] : 0.0f;
    }
    __syncthreads();
    for (int i = tid; i < 32 * K; i += kThreads) {
      const int r = i / K, k = i % K, b = s0 + r;
      xs[r][k] = b < batch ? Blob(fs[r][k / kBins], k % kBins) : 0.0f;
    }
    for (int i = tid; i < 32 * N; i += kThreads) {
      const int r = i / N, n = i % N, b = s0 + r;
      ds[r][n] = b < batch ? dz[static_cast<int64_t>(b) * N + n] : 0.0f;
    }
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < 32; ++r) {
      float a[T], d[T];
      LoadRow<T>(&xs[r][kg * T], a);
      LoadRow<T>(&ds[r][ng * T], d);
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) acc[i][j] += a[i] * d[j];
    }
    if (tid < N)
      for (int r = 0; r < 32; ++r) bacc += ds[r][tid];
    __syncthreads();
  }
  float *p = partial + static_cast<int64_t>(blockIdx.x) * kParams + layer_off;
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) p[(kg * T + i) * N + ng * T + j] = acc[i][j];
  if (tid < N) p[K * N + tid] = bacc;
}

__global__ void ReduceKernel(const float *partial, int chunks, float *grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  float s = 0.0f;
  for (int c = 0; c < chunks; ++c) s += partial[static_cast<int64_t>(c) * kParams + i];
  grad[i] = s;
}

// Adam (Kingma and Ba, 2015) with bias correction.
__global__ void AdamKernel(float *params, float *m, float *v, const float *grad, float lr, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  const float g = grad[i];
  const float mi = 0.9f * m[i] + 0.1f * g;
  const float vi = 0.999f * v[i] + 0.001f * g * g;
  m[i] = mi;
  v[i] = vi;
  params[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
}

// ---- sample gathering -----------------------------------------------------------------
__global__ void GatherKernel(const GuideSample *pool, uint64_t available, uint32_t cap, int batch, uint64_t seed,
                             float *features, float *dirs, float *weights) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= batch) return;
  const uint64_t valid = available < cap ? available : cap;
  Rng r(seed, 0, 0);
  r.ctr = make_uint4(static_cast<uint32_t>(i), 0x67617468u, static_cast<uint32_t>(seed >> 32), 0u);
  const uint64_t j = static_cast<uint64_t>(r.Next() * static_cast<float>(valid)) % (valid ? valid : 1);
  const GuideSample s = pool[j];
  float *f = features + static_cast<int64_t>(i) * kFeatures;
  f[0] = s.f0.x, f[1] = s.f0.y, f[2] = s.f0.z, f[3] = s.f0.w;
  f[4] = s.f1.x, f[5] = s.f1.y, f[6] = s.f1.z, f[7] = s.f1.w;
  dirs[3 * i] = s.dir_w.x, dirs[3 * i + 1] = s.dir_w.y, dirs[3 * i + 2] = s.dir_w.z;
  weights[i] = s.dir_w.w;
}

// Divides the weights by their mean (one block; fixed summation order).
// Training weights divided by their batch mean, in two deterministic passes:
// per-block sums in a fixed order, then every block forms the total from them.
constexpr int kSumBlocks = 256;

__global__ void __launch_bounds__(256) WeightSumKernel(const float *weights, int batch, double *part) {
  __shared__ double red[256];
  double s = 0.0;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < batch; i += kSumBlocks * 256) s += weights[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(256) WeightScaleKernel(float *weights, int batch, const double *part) {
  __shared__ float inv;
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int b = 0; b < kSumBlocks; ++b) total += part[b];
    const double mean = total / static_cast<double>(batch);
    inv = mean > 0.0 ? static_cast<float>(1.0 / mean) : 0.0f;
  }
  __syncthreads();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < batch; i += gridDim.x * 256) weights[i] *= inv;
}

inline unsigned Grid(int64_t n, int block) { return static_cast<unsigned>((n + block - 1) / block); }

}  // namespace

void LaunchGuidePack(const float *params, void *img, cudaStream_t st) {
  PackKernel<<<Grid(std::max(kImgChunks, kBiasFloats), 256), 256, 0, st>>>(params, static_cast<unsigned char *>(img));
}

void LaunchGuideInit(float *params, uint64_t seed, cudaStream_t st) {
  InitKernel<<<Grid(kParams, 256), 256, 0, st>>>(params, seed);
}

void LaunchGuideForward(const void *img, const float *features, int n, float *out, int32_t *status,
                        cudaStream_t st) {
  if (n <= 0) return;
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const unsigned grid = static_cast<unsigned>(std::max<int64_t>(
      1, std::min<int64_t>((static_cast<int64_t>(n) + kTcThreads - 1) / kTcThreads, std::max(sms, 1))));
  cudaFuncSetAttribute(ForwardKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemBytes);
  ForwardKernel<<<grid, kTcThreads, kTcSmemBytes, st>>>(img, features, n, out, status);
}

void LaunchGuideSample(const float *raw, int n, const float *u, float *mix, float *dirs, float *pdf,
                       cudaStream_t st) {
  if (n <= 0) return;
  MixKernel<<<Grid(n, 256), 256, 0, st>>>(raw, n, mix);
  SampleKernel<<<Grid(n, 256), 256, 0, st>>>(mix, n, u, dirs, pdf);
}

size_t GuideTrainBytes(int batch) {
  const size_t chunks = static_cast<size_t>(Chunks(batch));
  return sizeof(float) * (4ull * batch * kWidth + static_cast<size_t>(batch) * kOut + 2ull * batch * kWidth +
                          chunks * kParams + kParams) +
         sizeof(double) * (batch / kGuideLossSamples + 2 + kSumBlocks) + 256 * 10;
}

void GuideTrainCarve(void *base, int batch, GuideTrainBuffers *out) {
  char *p = static_cast<char *>(base);
  auto take = [&](size_t bytes) {
    char *r = p;
    p += (bytes + 255) / 256 * 256;
    return r;
  };
  out->h[0] = nullptr;
  for (int l = 1; l < 5; ++l) out->h[l] = reinterpret_cast<float *>(take(sizeof(float) * batch * kWidth));
  out->z = reinterpret_cast<float *>(take(sizeof(float) * batch * kOut));
  out->dz[0] = reinterpret_cast<float *>(take(sizeof(float) * batch * kWidth));
  out->dz[1] = reinterpret_cast<float *>(take(sizeof(float) * batch * kWidth));
  out->chunks = Chunks(batch);
  out->partial = reinterpret_cast<float *>(take(sizeof(float) * out->chunks * kParams));
  out->grad = reinterpret_cast<float *>(take(sizeof(float) * kParams));
  out->loss = reinterpret_cast<double *>(take(sizeof(double) * (batch / kGuideLossSamples + 2)));
  out->wsum = reinterpret_cast<double *>(take(sizeof(double) * kSumBlocks));
}

void LaunchGuideGradients(const float *params, const float *features, const float *dirs, const float *weights,
                          int batch, const GuideTrainBuffers &tb, cudaStream_t st) {
  const unsigned tiles = Grid(batch, kTile);
  auto W = [&](int l) { return params + MasterOffset(l); };
  auto B = [&](int l) { return params + MasterOffset(l) + In(l) * Out(l); };
  FwdLayerKernel<true, true><<<tiles, kTileThreads, 0, st>>>(features, W(0), B(0), kIn, tb.h[1], batch);
  for (int l = 1; l < 4; ++l)
    FwdLayerKernel<false, true><<<tiles, kTileThreads, 0, st>>>(tb.h[l], W(l), B(l), kWidth, tb.h[l + 1], batch);
  FwdLayerKernel<false, false><<<tiles, kTileThreads, 0, st>>>(tb.h[4], W(4), B(4), kWidth, tb.z, batch);
  LossKernel<<<Grid(batch, kGuideLossSamples), kThreads, 0, st>>>(tb.z, dirs, weights, batch, tb.loss);
  const unsigned chunks = static_cast<unsigned>(tb.chunks);
  const int chunk = ChunkSamples(batch);
  // layers 4..1: 64 x 64
  const float *dz = tb.z;
  int cur = 0;
  for (int l = 4; l >= 1; --l) {
    WgradSquareKernel<<<chunks, kThreads, 0, st>>>(tb.h[l], dz, batch, chunk, tb.partial, MasterOffset(l));
    BwdDataKernel<<<tiles, kTileThreads, 0, st>>>(dz, W(l), tb.h[l], tb.dz[cur], batch);
    dz = tb.dz[cur];
    cur ^= 1;
  }
  // layer 0: one-blob input, 256 x 64
  WgradBlobKernel<<<chunks, kThreads, 0, st>>>(features, dz, batch, chunk, tb.partial, MasterOffset(0));
  ReduceKernel<<<Grid(kParams, 256), 256, 0, st>>>(tb.partial, tb.chunks, tb.grad);
}

void LaunchGuideGather(const GuideSample *pool, uint64_t available, uint32_t cap, int batch, uint64_t seed,
                       float *features, float *dirs, float *weights, double *sums, cudaStream_t st) {
  GatherKernel<<<Grid(batch, 256), 256, 0, st>>>(pool, available, cap, batch, seed, features, dirs, weights);
  WeightSumKernel<<<kSumBlocks, 256, 0, st>>>(weights, batch, sums);
  WeightScaleKernel<<<std::max(1u, std::min(Grid(batch, 256), 1024u)), 256, 0, st>>>(weights, batch, sums);
}

void LaunchGuideAdam(float *params, float *m, float *v, const float *grad, float lr, int step, cudaStream_t st) {
  const float c1 = 1.0f - powf(0.9f, static_cast<float>(step));
  const float c2 = 1.0f - powf(0.999f, static_cast<float>(step));
  AdamKernel<<<Grid(kParams, 256), 256, 0, st>>>(params, m, v, grad, lr, c1, c2);
}

}  // namespace muon_gpu
