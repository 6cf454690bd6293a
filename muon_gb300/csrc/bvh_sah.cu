// BVH construction on the GPU with the host builder's binned SAH: the same
// split decisions as the top-down builder of scene_build.cc (32 centroid
// bins per axis, SAH with unit traversal and intersection costs, a leaf when
// a node of at most max_leaf references is no dearer as a leaf, the
// reference's BVH build replaced there as muon/acceleration.cc:204-458), so
// the tree has the host tree's nodes and boxes. Only the order of references
// inside a leaf and the node numbering differ: partitions here are stable,
// and interior nodes are numbered root first, then sibling pairs in the order
// of their parents' split positions.
//
// Every decision is taken with the same float operations as on the host,
// written with round-to-nearest intrinsics so that nothing is contracted into
// a fused multiply-add: centroid 0.5 (lo + hi), bin floor((c - lo) * 32 /
// extent), box areas, and the sweep's costs in the host's order. Bin
// contents (counts, min / max of boxes and centroids) are exact whatever the
// order in which references arrive.
//
// Three phases, queued by the host without waiting for any level: the lists'
// lengths stay on the device and are read back only where they can have run
// out.
//  * nodes of at least kSmallRefs references, level by level: a pass bins
//    the level's references into per-node bins (blocks of a chunk of
//    references accumulate in shared memory, then merge into global bins);
//    one warp per node sweeps the bins and decides; a stable partition
//    (per-chunk counts, per-node prefix, scatter) moves the references;
//  * smaller nodes, also level by level: a warp, or for the larger ones a
//    block, bins a node in shared memory, sweeps the bins with one lane per
//    bin, and partitions it with ballots;
//  * subtrees of at most kTinyRefs references, to their leaves: a lane per
//    reference, without bins.
//
// Every level is a handful of short kernels, bound by the latency of a
// node's chain (reference, box, bins, sweep) and not by bandwidth: a scene of
// 87 k triangles opens in 1.6 ms, one of 1.3 M in 8.2 ms. With a host that
// waited for each level, one warp per small node down to the leaves, and
// atomics per node on the lists' lengths, these were 2.5 and 12.4 ms.
//
// A node's box and its children's centroid bounds come from its bins. A node
// writes its own box and link into its parent's child slot, and an interior
// node keeps its entry at index (split position - 1) of a sparse array; a
// scan of the entries' interior-child counts gives the dense numbering at
// the end, siblings side by side.
#include <cub/device/device_scan.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bvh_build.h"

namespace muon_gpu {

namespace {

constexpr int kSahBins = 32;
// Words of one bin: reference count, box lo / hi, centroid lo / hi (floats
// as order-preserving keys).
constexpr int kBinWords = 13;
constexpr int kNodeBinWords = 3 * kSahBins * kBinWords;
constexpr int kSmallRefs = 2048;
// References per block of the level phase: the largest chunk, and the
// smallest one (ChunkRefs).
constexpr int kLevelThreads = 256;
constexpr int kMaxChunk = 8 * kLevelThreads, kMinChunk = kLevelThreads;
constexpr int kPerThread = kMaxChunk / kLevelThreads;
constexpr int kPlanThreads = 1024;
constexpr int kMaxLevels = 64;
constexpr int kSmallWarps = 8;
// Blocks per SM: two keep the kernel's 118 registers out of memory; three
// to five (80 to 48 registers, spilled) measure alike or 1% slower.
constexpr int kSmallBlocks = 2;
// Small nodes of at least this many references are taken by a whole block
// (a warp took 120 us for a first level of nodes near kSmallRefs, a block
// takes 25; lines from 64 to 1,024 measure alike).
constexpr int kTeamRefs = 256;
constexpr int kTeamPer = kSmallRefs / (kSmallWarps * 32);
// Nodes of at most this many references are built to their leaves by as many
// lanes (a power of two). A scene of 1.3 M triangles opens in 8.2 ms so, in
// 8.5 with 4, 8.3 with 16, 8.7 with 32 and 10.4 with none.
constexpr int kTinyRefs = 8;
constexpr int kTinyWarps = 4;
// Children a warp keeps before it appends them to the next level's list.
constexpr int kKids = 16;
// levels between checks of the lists' lengths once they may have run out,
// and small-node levels at most
constexpr int kLevelsPerCheck = 3;
constexpr int kMaxSmallLevels = 4096;

// Chunk of a build of n references: two blocks per SM in the level phase
// where n allows it, since a block's time is its references' chain of shared
// atomics, but no smaller, since each block merges 1,248 words into the
// node's bins.
int ChunkRefs(int n, int sms) {
  int chunk = kMinChunk;
  while (chunk < kMaxChunk && n / chunk > 2 * sms) chunk *= 2;
  return chunk;
}

inline unsigned Blocks(int64_t n, int threads) { return static_cast<unsigned>((n + threads - 1) / threads); }

__device__ __forceinline__ unsigned FloatKey(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float KeyFloat(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// A node waiting to be split: its references idx[start, end), the child slot
// of its parent it fills (sparse index * 2 + slot) and its centroid bounds.
struct PendingNode {
  int32_t start, end, parent, depth;
  float clo[3], chi[3];
};

// How a level node was split: axis >= 0 binned SAH at `bin`; -1 leaf; -2 the
// first half by position (every centroid coincides).
struct Decision {
  int32_t axis, bin, mid, pad;
  float lo, scale;
};

struct SahStats {
  unsigned long long leaves;
  int max_depth, max_leaf, root, error;
  int level_count[2], work_count;  // lengths of the level lists and of the level's work
  int small_count[3], tiny_count;  // lengths of the small-node lists (in turn) and of the tiny one
  int nodes;
};

// What the nodes that a warp (or thread) decided add to SahStats.
struct NodeStats {
  int leaves = 0, max_depth = 0, max_leaf = 0;
};

__device__ __forceinline__ float Centroid(float lo, float hi) { return __fmul_rn(0.5f, __fadd_rn(lo, hi)); }

// scale_axis as the host builder forms it: kBins / extent, 0 for no extent.
__device__ __forceinline__ float BinScale(float lo, float hi) {
  const float extent = __fsub_rn(hi, lo);
  return extent > 0.0f ? __fdiv_rn(static_cast<float>(kSahBins), extent) : 0.0f;
}
__device__ __forceinline__ int BinOf(float c, float lo, float scale) {
  const int k = __float2int_rz(__fmul_rn(__fsub_rn(c, lo), scale));
  return max(0, min(kSahBins - 1, k));
}

// Area of a box as the host builder computes it (0 for an empty box).
__device__ __forceinline__ float BoxArea(const float *lo, const float *hi) {
  const float dx = __fsub_rn(hi[0], lo[0]), dy = __fsub_rn(hi[1], lo[1]), dz = __fsub_rn(hi[2], lo[2]);
  if (!(dx >= 0.0f) || !(dy >= 0.0f) || !(dz >= 0.0f)) return 0.0f;
  return __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dx, dz)), __fmul_rn(dy, dz)));
}

__device__ __forceinline__ void LoadRef(const float4 *box8, int ref, float *lo, float *hi) {
  const float4 a = __ldg(box8 + 2 * ref), b = __ldg(box8 + 2 * ref + 1);
  lo[0] = a.x, lo[1] = a.y, lo[2] = a.z;
  hi[0] = b.x, hi[1] = b.y, hi[2] = b.z;
}

// Empty bins: count 0; lower bounds start at the largest key, upper bounds
// at 0. One thread per bin (13 words apart: no bank conflict).
__device__ __forceinline__ void InitBins(uint32_t *bins, int i0, int step) {
  for (int b = i0; b < 3 * kSahBins; b += step) {
    for (int f = 0; f < kBinWords; ++f)
      bins[b * kBinWords + f] = (f >= 1 && f <= 3) || (f >= 7 && f <= 9) ? 0xffffffffu : 0u;
  }
}

// The bins of m nodes, thread i0 of `step` threads.
__device__ __forceinline__ void InitBinsOf(uint32_t *bins, int m, int64_t i0, int64_t step) {
  for (int64_t w = i0; w < static_cast<int64_t>(m) * kNodeBinWords; w += step) {
    const int f = static_cast<int>(w % kBinWords);
    bins[w] = (f >= 1 && f <= 3) || (f >= 7 && f <= 9) ? 0xffffffffu : 0u;
  }
}

// Adds one reference to a node's bins (shared or global memory).
__device__ __forceinline__ void BinRef(uint32_t *bins, const float *lo, const float *hi, const float *clo,
                                       const float *scale) {
  float c[3];
  for (int k = 0; k < 3; ++k) c[k] = Centroid(lo[k], hi[k]);
  for (int axis = 0; axis < 3; ++axis) {
    uint32_t *b = bins + (axis * kSahBins + BinOf(c[axis], clo[axis], scale[axis])) * kBinWords;
    atomicAdd(b, 1u);
    for (int k = 0; k < 3; ++k) {
      atomicMin(b + 1 + k, FloatKey(lo[k]));
      atomicMax(b + 4 + k, FloatKey(hi[k]));
      atomicMin(b + 7 + k, FloatKey(c[k]));
      atomicMax(b + 10 + k, FloatKey(c[k]));
    }
  }
}

// Merges shared bins into global ones (bins that received nothing are
// skipped).
__device__ __forceinline__ void FlushBins(const uint32_t *s, uint32_t *g, int i0, int step) {
  for (int w = i0; w < kNodeBinWords; w += step) {
    const int f = w % kBinWords;
    if (s[w - f] == 0) continue;
    if (f == 0) atomicAdd(g + w, s[w]);
    else if ((f >= 1 && f <= 3) || (f >= 7 && f <= 9)) atomicMin(g + w, s[w]);
    else atomicMax(g + w, s[w]);
  }
}

// A node's box and split, from its bins; the same in every lane of the warp.
struct NodeSplit {
  float lo[3], hi[3];  // the node's box
  int axis, bin;       // Decision::axis / bin
  int left_n;          // references that go left
  float lclo[3], lchi[3], rclo[3], rchi[3];  // the children's centroid bounds
};

__device__ __forceinline__ float WarpMin(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float WarpMax(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ int WarpSum(int v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// SplitSah's two sweeps over one axis (scene_build.cc), lane b holding bin
// b: the right sweep's box of bins b..31 and the left sweep's box of bins
// 0..b are unions (exact in any order), so suffix and prefix scans across
// the lanes give the host's boxes, areas and costs; the cheapest split of the
// axis, the first bin at the minimum, in every lane; bin -1 when none leaves
// both sides non-empty.
__device__ void SweepAxis(const uint32_t *ab, int lane, float *best_cost, int *best_bin) {
  const uint32_t *x = ab + lane * kBinWords;
  const int c = static_cast<int>(x[0]);
  float blo[3], bhi[3];
  for (int k = 0; k < 3; ++k) {
    blo[k] = c ? KeyFloat(x[1 + k]) : INFINITY;
    bhi[k] = c ? KeyFloat(x[4 + k]) : -INFINITY;
  }
  float llo[3], lhi[3], rlo[3], rhi[3];
  int ln = c, rn = c;
  for (int k = 0; k < 3; ++k) llo[k] = rlo[k] = blo[k], lhi[k] = rhi[k] = bhi[k];
  for (int o = 1; o < kSahBins; o <<= 1) {
    const int up_n = __shfl_up_sync(0xffffffffu, ln, o), down_n = __shfl_down_sync(0xffffffffu, rn, o);
    if (lane >= o) ln += up_n;
    if (lane + o < kSahBins) rn += down_n;
    for (int k = 0; k < 3; ++k) {
      const float ul = __shfl_up_sync(0xffffffffu, llo[k], o), uh = __shfl_up_sync(0xffffffffu, lhi[k], o);
      const float dl = __shfl_down_sync(0xffffffffu, rlo[k], o), dh = __shfl_down_sync(0xffffffffu, rhi[k], o);
      if (lane >= o) llo[k] = fminf(llo[k], ul), lhi[k] = fmaxf(lhi[k], uh);
      if (lane + o < kSahBins) rlo[k] = fminf(rlo[k], dl), rhi[k] = fmaxf(rhi[k], dh);
    }
  }
  // the right side of split b is bins b+1..31
  const float right_area = __shfl_down_sync(0xffffffffu, BoxArea(rlo, rhi), 1);
  const int right_n = __shfl_down_sync(0xffffffffu, rn, 1);
  float cost = INFINITY;
  if (lane < kSahBins - 1 && ln != 0 && right_n != 0)
    cost = __fadd_rn(__fmul_rn(BoxArea(llo, lhi), __int2float_rn(ln)),
                     __fmul_rn(right_area, __int2float_rn(right_n)));
  int bin = cost < INFINITY ? lane : kSahBins;
  for (int o = 16; o > 0; o >>= 1) {
    const float oc = __shfl_xor_sync(0xffffffffu, cost, o);
    const int ob = __shfl_xor_sync(0xffffffffu, bin, o);
    if (oc < cost || (oc == cost && ob < bin)) cost = oc, bin = ob;
  }
  *best_cost = cost;
  *best_bin = bin < kSahBins ? bin : -1;
}

// Leaf (-1), split along the cheapest axis (>= 0), or halves by position
// (-2, no axis separates the references), as in Builder::Build.
__device__ __forceinline__ int DecideAxis(int n, int max_leaf, int best_axis, float best_cost, const float *lo,
                                          const float *hi) {
  if (best_axis < 0) return n <= max_leaf ? -1 : -2;
  const float parent_area = BoxArea(lo, hi);
  const float split_cost = __fadd_rn(1.0f, __fdiv_rn(__fmul_rn(1.0f, best_cost), fmaxf(parent_area, 1e-30f)));
  const float leaf_cost = __fmul_rn(1.0f, __int2float_rn(n));
  return (n <= max_leaf && leaf_cost <= split_cost) ? -1 : best_axis;
}

// Evaluates a node of n >= 2 references from its bins (all 32 lanes call;
// lane b reads bin b). Decision as in Builder::Build / SplitSah.
__device__ NodeSplit EvaluateNode(const uint32_t *bins, const PendingNode &nd, int max_leaf, int lane) {
  NodeSplit s;
  const int n = nd.end - nd.start;
  {
    // the node box: the union of every bin of axis 0
    const uint32_t *x = bins + lane * kBinWords;
    const bool full = x[0] != 0u;
    for (int k = 0; k < 3; ++k) {
      s.lo[k] = WarpMin(full ? KeyFloat(x[1 + k]) : INFINITY);
      s.hi[k] = WarpMax(full ? KeyFloat(x[4 + k]) : -INFINITY);
    }
  }
  float best_cost = INFINITY;
  int best_axis = -1, best_bin = -1;
  for (int a = 0; a < 3; ++a) {
    if (!(__fsub_rn(nd.chi[a], nd.clo[a]) > 0.0f)) continue;
    float c;
    int b;
    SweepAxis(bins + a * kSahBins * kBinWords, lane, &c, &b);
    if (b >= 0 && c < best_cost) best_cost = c, best_axis = a, best_bin = b;
  }
  s.bin = best_bin;
  s.axis = DecideAxis(n, max_leaf, best_axis, best_cost, s.lo, s.hi);
  if (s.axis >= 0) {
    const uint32_t *x = bins + (s.axis * kSahBins + lane) * kBinWords;
    const bool full = x[0] != 0u, left = lane <= s.bin;
    s.left_n = WarpSum(left ? static_cast<int>(x[0]) : 0);
    for (int k = 0; k < 3; ++k) {
      const float cl = full ? KeyFloat(x[7 + k]) : INFINITY, ch = full ? KeyFloat(x[10 + k]) : -INFINITY;
      s.lclo[k] = WarpMin(left ? cl : INFINITY);
      s.lchi[k] = WarpMax(left ? ch : -INFINITY);
      s.rclo[k] = WarpMin(left ? INFINITY : cl);
      s.rchi[k] = WarpMax(left ? -INFINITY : ch);
    }
  } else {
    // a leaf, or halves by position when every centroid coincides (the
    // halves keep the node's centroid bounds)
    s.left_n = n / 2;
    for (int k = 0; k < 3; ++k) s.lclo[k] = s.rclo[k] = nd.clo[k], s.lchi[k] = s.rchi[k] = nd.chi[k];
  }
  return s;
}

// Writes a child's padded box and link into slot (parent & 1) of sparse
// entry parent >> 1 (the padding of the host builder's Pad).
__device__ void WriteSlot(BvhNode *sparse, int parent, const float *lo, const float *hi, int link) {
  float plo[3], phi[3];
  for (int k = 0; k < 3; ++k) {
    if (!(lo[k] <= hi[k])) {
      plo[k] = lo[k], phi[k] = hi[k];
      continue;
    }
    const float m = __fadd_rn(fmaxf(fabsf(lo[k]), fabsf(hi[k])), __fsub_rn(hi[k], lo[k]));
    const float e = __fadd_rn(__fmul_rn(m, 4e-7f), 1e-30f);
    plo[k] = __fsub_rn(lo[k], e);
    phi[k] = __fadd_rn(hi[k], e);
  }
  BvhNode &nd = sparse[parent >> 1];
  if ((parent & 1) == 0) {
    nd.a = F4{plo[0], phi[0], plo[1], phi[1]};
    nd.c.x = plo[2], nd.c.y = phi[2];
    nd.d.x = link;
  } else {
    nd.b = F4{plo[0], phi[0], plo[1], phi[1]};
    nd.c.z = plo[2], nd.c.w = phi[2];
    nd.d.y = link;
  }
}

// Lane 0: records a decided node (leaf or interior) and returns the
// children to build (false for a leaf).
__device__ bool EmitNode(const PendingNode &nd, const NodeSplit &s, BvhNode *sparse, int *used, uint8_t *last,
                         NodeStats *ns, PendingNode *left, PendingNode *right) {
  ns->max_depth = max(ns->max_depth, nd.depth);
  if (s.axis == -1) {
    WriteSlot(sparse, nd.parent, s.lo, s.hi, ~nd.start);
    last[nd.end - 1] = 1;
    ns->leaves += 1;
    ns->max_leaf = max(ns->max_leaf, nd.end - nd.start);
    return false;
  }
  const int mid = nd.start + s.left_n;
  const int p = mid - 1;
  used[p] = 1;
  WriteSlot(sparse, nd.parent, s.lo, s.hi, p);
  *left = PendingNode{nd.start, mid, 2 * p, nd.depth + 1, {s.lclo[0], s.lclo[1], s.lclo[2]},
                      {s.lchi[0], s.lchi[1], s.lchi[2]}};
  *right = PendingNode{mid, nd.end, 2 * p + 1, nd.depth + 1, {s.rclo[0], s.rclo[1], s.rclo[2]},
                       {s.rchi[0], s.rchi[1], s.rchi[2]}};
  return true;
}

__device__ __forceinline__ Decision MakeDecision(const PendingNode &nd, const NodeSplit &s) {
  Decision d{};
  d.axis = s.axis;
  d.bin = s.bin;
  d.mid = nd.start + s.left_n;
  if (s.axis >= 0) {
    d.lo = nd.clo[s.axis];
    d.scale = BinScale(nd.clo[s.axis], nd.chi[s.axis]);
  }
  return d;
}

__device__ __forceinline__ void AddStats(const NodeStats &ns, SahStats *st) {
  if (ns.max_depth) atomicMax(&st->max_depth, ns.max_depth);
  if (ns.leaves) atomicAdd(&st->leaves, static_cast<unsigned long long>(ns.leaves));
  if (ns.max_leaf) atomicMax(&st->max_leaf, ns.max_leaf);
}

// Whether reference `ref` goes to the left child (false for a value that is
// not a reference; the binning pass flags those).
__device__ __forceinline__ bool GoesLeft(const Decision &d, const float4 *box8, int n, int ref) {
  if (static_cast<unsigned>(ref) >= static_cast<unsigned>(n)) return false;
  const float4 a = __ldg(box8 + 2 * ref), b = __ldg(box8 + 2 * ref + 1);
  const float lo = d.axis == 0 ? a.x : (d.axis == 1 ? a.y : a.z);
  const float hi = d.axis == 0 ? b.x : (d.axis == 1 ? b.y : b.z);
  return BinOf(Centroid(lo, hi), d.lo, d.scale) <= d.bin;
}

// Boxes into two float4s per reference, the identity reference order, and
// the root's centroid bounds (order-preserving keys, min then max).
__global__ void PackKernel(const float *boxes, int n, float4 *box8, int32_t *idx, unsigned *cbounds) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  __shared__ unsigned sb[6];  // the block's bounds: six global atomics per block
  if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
  __syncthreads();
  unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  if (i < n) {
    const float *b = boxes + 6 * static_cast<int64_t>(i);
    box8[2 * i] = make_float4(b[0], b[1], b[2], 0.0f);
    box8[2 * i + 1] = make_float4(b[3], b[4], b[5], 0.0f);
    idx[i] = i;
    for (int k = 0; k < 3; ++k) lo[k] = hi[k] = FloatKey(Centroid(b[k], b[3 + k]));
  }
  for (int k = 0; k < 3; ++k) {
    lo[k] = __reduce_min_sync(0xffffffffu, lo[k]);
    hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
  }
  if ((threadIdx.x & 31) == 0) {
    for (int k = 0; k < 3; ++k) atomicMin(sb + k, lo[k]), atomicMax(sb + 3 + k, hi[k]);
  }
  __syncthreads();
  if (threadIdx.x < 3) atomicMin(cbounds + threadIdx.x, sb[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(cbounds + threadIdx.x, sb[threadIdx.x]);
}

// The root as a pending node: all references, the virtual parent slot
// (sparse entry n - 1), its centroid bounds; into the level list or, when it
// is small, the small list.
__global__ void RootKernel(int n, const unsigned *cbounds, PendingNode *level, PendingNode *small, PendingNode *tiny,
                           SahStats *st) {
  PendingNode r{};
  r.start = 0;
  r.end = n;
  r.parent = 2 * (n - 1);
  r.depth = 0;
  for (int k = 0; k < 3; ++k) r.clo[k] = KeyFloat(cbounds[k]), r.chi[k] = KeyFloat(cbounds[3 + k]);
  if (n >= kSmallRefs) {
    level[0] = r;
    st->level_count[0] = 1;
  } else if (n <= kTinyRefs) {
    tiny[0] = r;
    st->tiny_count = 1;
  } else {
    small[0] = r;
    st->small_count[0] = 1;
  }
}

// Exclusive scan of one int per thread over a block of kThreads threads (all
// call); returns the thread's prefix and sets *total.
template <int kThreads>
__device__ int BlockExclusiveScan(int v, int *total) {
  __shared__ int warp_sums[kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  int before = 0, all = 0;
  for (int k = 0; k < kThreads / 32; ++k) {
    const int s = warp_sums[k];
    if (k < w) before += s;
    all += s;
  }
  __syncthreads();
  *total = all;
  return before + x - v;
}

__device__ __forceinline__ int LevelNodes(const SahStats *st, int cur, int cap) { return min(st->level_count[cur], cap); }

// Opens a level: block 0 lists its work, one item (node, first reference)
// per chunk of every node, and each node's first item (first[j], j <= m);
// the other blocks empty the nodes' bins. The counts stay on the device, so
// the host queues the levels without waiting for any; kernels of a level are
// launched for as many nodes and items as there can be and leave at once
// where there are none.
__global__ void __launch_bounds__(kPlanThreads) LevelPlanKernel(const PendingNode *level, int cap, int cur, int chunk,
                                                                int work_cap, int2 *work, int *first, uint32_t *bins,
                                                                SahStats *st) {
  const int m = LevelNodes(st, cur, cap);
  if (blockIdx.x > 0) {
    const int stride = (gridDim.x - 1) * kPlanThreads;
    InitBinsOf(bins, m, (blockIdx.x - 1) * kPlanThreads + threadIdx.x, stride);
    return;
  }
  int items = 0;
  for (int base = 0; base < m; base += kPlanThreads) {
    const int j = base + threadIdx.x;
    int c = 0, start = 0;
    if (j < m) {
      start = level[j].start;
      c = (level[j].end - start + chunk - 1) / chunk;
    }
    int total = 0;
    const int at = items + BlockExclusiveScan<kPlanThreads>(c, &total);
    if (j < m) first[j] = at;
    items += total;
  }
  if (threadIdx.x == 0) {
    first[m] = items;
    st->level_count[cur ^ 1] = 0;
    st->work_count = min(items, work_cap);
    if (items > work_cap) atomicExch(&st->error, 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < min(items, work_cap); i += kPlanThreads) {
    int lo = 0, hi = m - 1;  // the last node whose first item is at most i
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (first[mid] <= i) lo = mid;
      else hi = mid - 1;
    }
    work[i] = make_int2(lo, level[lo].start + (i - first[lo]) * chunk);
  }
}

// One block per work item (level node, chunk of references).
__global__ void __launch_bounds__(kLevelThreads) LevelBinKernel(const float4 *box8, const int32_t *idx, int n,
                                                                 int chunk, const PendingNode *level,
                                                                 const int2 *work, uint32_t *bins, SahStats *st) {
  __shared__ uint32_t sb[kNodeBinWords];
  if (static_cast<int>(blockIdx.x) >= st->work_count) return;
  const int2 w = work[blockIdx.x];
  const PendingNode nd = level[w.x];
  InitBins(sb, threadIdx.x, kLevelThreads);
  float scale[3];
  for (int k = 0; k < 3; ++k) scale[k] = BinScale(nd.clo[k], nd.chi[k]);
  __syncthreads();
  const int end = min(w.y + chunk, nd.end);
  for (int i = w.y + threadIdx.x; i < end; i += kLevelThreads) {
    const int ref = idx[i];
    if (static_cast<unsigned>(ref) >= static_cast<unsigned>(n)) {
      atomicExch(&st->error, 5);  // not a reference: the partition went wrong
      continue;
    }
    float lo[3], hi[3];
    LoadRef(box8, ref, lo, hi);
    BinRef(sb, lo, hi, nd.clo, scale);
  }
  __syncthreads();
  FlushBins(sb, bins + static_cast<int64_t>(w.x) * kNodeBinWords, threadIdx.x, kLevelThreads);
}

// One warp per level node: decide, record, queue the children.
__global__ void LevelSplitKernel(const PendingNode *level, int cur, const uint32_t *bins, int max_leaf, Decision *dec,
                                 BvhNode *sparse, int *used, uint8_t *last, PendingNode *next, int next_cap,
                                 PendingNode *small, int small_cap, PendingNode *tiny, int tiny_cap,
                                 SahStats *st) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= LevelNodes(st, cur, next_cap)) return;
  const PendingNode nd = level[warp];
  const NodeSplit s = EvaluateNode(bins + static_cast<int64_t>(warp) * kNodeBinWords, nd, max_leaf, lane);
  if (lane != 0) return;
  dec[warp] = MakeDecision(nd, s);
  PendingNode kids[2];
  NodeStats ns;
  const bool split = EmitNode(nd, s, sparse, used, last, &ns, &kids[0], &kids[1]);
  AddStats(ns, st);
  if (!split) return;
  for (const PendingNode &k : kids) {
    if (k.end - k.start >= kSmallRefs) {
      const int at = atomicAdd(&st->level_count[cur ^ 1], 1);
      if (at < next_cap) next[at] = k;
      else atomicExch(&st->error, 2);
    } else if (k.end - k.start <= kTinyRefs) {
      const int at = atomicAdd(&st->tiny_count, 1);
      if (at < tiny_cap) tiny[at] = k;
      else atomicExch(&st->error, 3);
    } else {
      const int at = atomicAdd(&st->small_count[0], 1);
      if (at < small_cap) small[at] = k;
      else atomicExch(&st->error, 3);
    }
  }
}

// References that go left in each work item's chunk.
__global__ void __launch_bounds__(kLevelThreads) LevelCountKernel(const float4 *box8, const int32_t *idx, int n,
                                                                   int chunk, const PendingNode *level,
                                                                   const Decision *dec, const int2 *work,
                                                                   int *chunk_left, const SahStats *st) {
  if (static_cast<int>(blockIdx.x) >= st->work_count) return;
  const int2 w = work[blockIdx.x];
  const Decision d = dec[w.x];
  if (d.axis < 0) return;
  const int end = min(w.y + chunk, level[w.x].end);
  int c = 0;
  for (int i = w.y + threadIdx.x; i < end; i += kLevelThreads) c += GoesLeft(d, box8, n, idx[i]) ? 1 : 0;
  int total = 0;
  BlockExclusiveScan<kLevelThreads>(c, &total);
  if (threadIdx.x == 0) chunk_left[blockIdx.x] = total;
}

// Per level node (one block each), the exclusive prefix of its chunks' left
// counts (its work items are first[j] .. first[j + 1] - 1).
__global__ void __launch_bounds__(kLevelThreads) LevelScanKernel(const Decision *dec, int cur, int cap,
                                                                 const int *first, int *chunk_left,
                                                                 const SahStats *st) {
  const int j = blockIdx.x;
  if (j >= LevelNodes(st, cur, cap) || dec[j].axis < 0) return;
  const int end = min(first[j + 1], st->work_count);
  int acc = 0;
  for (int base = first[j]; base < end; base += kLevelThreads) {
    const int w = base + threadIdx.x;
    int total = 0;
    const int before = BlockExclusiveScan<kLevelThreads>(w < end ? chunk_left[w] : 0, &total);
    if (w < end) chunk_left[w] = acc + before;
    acc += total;
  }
}

// Stable partition of each chunk into tmp: thread t holds references
// [w.y + per t, + per); left and right counts packed in one
// scan (a chunk holds fewer than 65,536 references).
__global__ void __launch_bounds__(kLevelThreads) LevelScatterKernel(const float4 *box8, const int32_t *idx, int n,
                                                                     int chunk, int32_t *tmp,
                                                                     const PendingNode *level, const Decision *dec,
                                                                     const int2 *work, const int *chunk_left,
                                                                     SahStats *st) {
  if (static_cast<int>(blockIdx.x) >= st->work_count) return;
  const int2 w = work[blockIdx.x];
  const Decision d = dec[w.x];
  if (d.axis < 0) return;
  const PendingNode nd = level[w.x];
  const int end = min(w.y + chunk, nd.end);
  const int per = chunk / kLevelThreads;
  const int i0 = w.y + threadIdx.x * per;
  int ref[kPerThread];
  unsigned left_mask = 0;
  int nl = 0, nr = 0;
  for (int k = 0; k < kPerThread; ++k) {
    const int i = i0 + k;
    ref[k] = -1;
    if (k < per && i < end) {
      ref[k] = idx[i];
      if (GoesLeft(d, box8, n, ref[k])) left_mask |= 1u << k, ++nl;
      else ++nr;
    }
  }
  int total = 0;
  const int before = BlockExclusiveScan<kLevelThreads>(nl | (nr << 16), &total);
  int l = nd.start + chunk_left[blockIdx.x] + (before & 0xffff);
  int r = d.mid + (w.y - nd.start - chunk_left[blockIdx.x]) + (before >> 16);
  for (int k = 0; k < kPerThread; ++k) {
    if (ref[k] < 0) continue;
    const bool left = (left_mask & (1u << k)) != 0;
    const int at = left ? l++ : r++;
    if (left ? (at < nd.start || at >= d.mid) : (at < d.mid || at >= nd.end)) {
      atomicExch(&st->error, 6);  // the counts and the bins disagree
      continue;
    }
    tmp[at] = ref[k];
  }
}

__global__ void __launch_bounds__(kLevelThreads) LevelCopyKernel(int32_t *idx, const int32_t *tmp, int chunk,
                                                                  const PendingNode *level, const Decision *dec,
                                                                  const int2 *work, const SahStats *st) {
  if (static_cast<int>(blockIdx.x) >= st->work_count) return;
  const int2 w = work[blockIdx.x];
  if (dec[w.x].axis < 0) return;
  const int end = min(w.y + chunk, level[w.x].end);
  for (int i = w.y + threadIdx.x; i < end; i += kLevelThreads) idx[i] = tmp[i];
}

// Shared memory of SmallLevelKernel.
struct SmallShared {
  uint32_t bins[kSmallWarps][kNodeBinWords];
  PendingNode kids[kSmallWarps][kKids];
  Decision dec;
  int left[kSmallWarps], split;
  int kid_count[2][kSmallWarps], kid_base[2];
  int leaves, max_depth, max_leaf;
};

// A pending node's references as they stand, in the lists' bounds.
__device__ __forceinline__ bool ValidNode(const PendingNode &nd, int n_refs) {
  return nd.end > nd.start && nd.start >= 0 && nd.end <= n_refs;
}

// The lists that a level's children go to: the next level's and the tiny one.
struct KidLists {
  PendingNode *list[2];
  int cap[2];
  int *count[2];
};

// Stores lane's child into list `kind` at the place that follows from the
// list's first free place.
__device__ __forceinline__ void StoreKid(const KidLists &o, const PendingNode &k, int kind, int at, SahStats *st) {
  if (at < o.cap[kind]) o.list[kind][at] = k;
  else atomicExch(&st->error, 3);
}

// Appends the `count` children that a warp keeps to their lists.
__device__ __forceinline__ void FlushKids(const PendingNode *kids, int count, const KidLists &o, int lane,
                                          SahStats *st) {
  __syncwarp();
  const bool have = lane < count;
  const bool tiny = have && kids[lane].end - kids[lane].start <= kTinyRefs;
  const unsigned in[2] = {__ballot_sync(0xffffffffu, have && !tiny), __ballot_sync(0xffffffffu, tiny)};
  int base = 0;
  if (lane < 2 && in[lane]) base = atomicAdd(o.count[lane], __popc(in[lane]));
  base = __shfl_sync(0xffffffffu, base, tiny ? 1 : 0);
  if (have) StoreKid(o, kids[lane], tiny, base + __popc(in[tiny] & ((1u << lane) - 1u)), st);
  __syncwarp();
}

// One small node by the whole block (2 <= references <= kSmallRefs): each
// warp holds a contiguous part of the references in registers, bins them,
// warp 0 decides, and the parts' left counts give every warp its places.
__device__ void TeamNode(SmallShared &sh, const PendingNode &nd, const float4 *box8, int32_t *idx, int n_refs,
                         int max_leaf, BvhNode *sparse, int *used, uint8_t *last, NodeStats *ns,
                         int *kid_count, SahStats *st) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t *bins = sh.bins[0];
  __syncthreads();  // the warps' own bins and the previous node's values have been read
  InitBins(bins, threadIdx.x, kSmallWarps * 32);
  const int n = nd.end - nd.start;
  const int part = (n + kSmallWarps * 32 - 1) / (kSmallWarps * 32) * 32;  // references per warp
  const int p0 = nd.start + wid * part, p1 = min(p0 + part, nd.end);
  int ref[kTeamPer];
#pragma unroll
  for (int k = 0; k < kTeamPer; ++k) {
    const int i = p0 + 32 * k + lane;
    ref[k] = i < p1 ? idx[i] : -1;
  }
  float scale[3];
  for (int k = 0; k < 3; ++k) scale[k] = BinScale(nd.clo[k], nd.chi[k]);
  __syncthreads();
  bool bad = false;
#pragma unroll
  for (int k = 0; k < kTeamPer; ++k) {
    if (p0 + 32 * k + lane >= p1) continue;
    if (static_cast<unsigned>(ref[k]) >= static_cast<unsigned>(n_refs)) {
      bad = true;
      continue;
    }
    float lo[3], hi[3];
    LoadRef(box8, ref[k], lo, hi);
    BinRef(bins, lo, hi, nd.clo, scale);
  }
  if (__syncthreads_or(bad)) {
    if (threadIdx.x == 0) atomicExch(&st->error, 5);
    return;
  }
  if (wid == 0) {
    const NodeSplit s = EvaluateNode(bins, nd, max_leaf, lane);
    if (lane == 0) {
      sh.split = EmitNode(nd, s, sparse, used, last, ns, &sh.kids[0][*kid_count], &sh.kids[0][*kid_count + 1]);
      sh.dec = MakeDecision(nd, s);
    }
  }
  __syncthreads();
  if (wid == 0 && sh.split) *kid_count += 2;
  const Decision d = sh.dec;
  if (!sh.split || d.axis < 0) return;
  unsigned left[kTeamPer];
  int nl = 0;
#pragma unroll
  for (int k = 0; k < kTeamPer; ++k) {
    left[k] = __ballot_sync(0xffffffffu, p0 + 32 * k + lane < p1 && GoesLeft(d, box8, n_refs, ref[k]));
    nl += __popc(left[k]);
  }
  if (lane == 0) sh.left[wid] = nl;
  __syncthreads();  // every reference has been read
  int l = nd.start, r = d.mid + (p0 - nd.start);
  for (int w = 0; w < wid; ++w) l += sh.left[w], r -= sh.left[w];
#pragma unroll
  for (int k = 0; k < kTeamPer; ++k) {
    const int i = p0 + 32 * k + lane;
    const unsigned valid = __ballot_sync(0xffffffffu, i < p1);
    if (i < p1) {
      const bool go = (left[k] >> lane) & 1u;
      const int at = go ? l + __popc(left[k] & lt) : r + __popc(valid & ~left[k] & lt);
      if (at >= (go ? nd.start : d.mid) && at < (go ? d.mid : nd.end)) idx[at] = ref[k];
      else atomicExch(&st->error, 6);
    }
    l += __popc(left[k]);
    r += __popc(valid & ~left[k]);
  }
}

// One small node of n >= 2 references by a warp.
__device__ void WarpNode(uint32_t *bins, PendingNode *kids, int *kid_count, const PendingNode &nd, const float4 *box8,
                         int32_t *idx, int32_t *tmp, int n_refs, int max_leaf, BvhNode *sparse, int *used,
                         uint8_t *last, NodeStats *ns, int lane, SahStats *st) {
  const unsigned lt = (1u << lane) - 1u;
  __syncwarp();  // the previous node's bins have been read
  InitBins(bins, lane, 32);
  float scale[3];
  for (int k = 0; k < 3; ++k) scale[k] = BinScale(nd.clo[k], nd.chi[k]);
  __syncwarp();
  bool bad = false;
#pragma unroll 2
  for (int i = nd.start + lane; i < nd.end; i += 32) {
    const int ref = idx[i];
    if (static_cast<unsigned>(ref) >= static_cast<unsigned>(n_refs)) {
      bad = true;
      continue;
    }
    float lo[3], hi[3];
    LoadRef(box8, ref, lo, hi);
    BinRef(bins, lo, hi, nd.clo, scale);
  }
  if (__any_sync(0xffffffffu, bad)) {
    if (lane == 0) atomicExch(&st->error, 5);
    return;
  }
  __syncwarp();
  const NodeSplit s = EvaluateNode(bins, nd, max_leaf, lane);
  bool split = false;
  if (lane == 0) split = EmitNode(nd, s, sparse, used, last, ns, &kids[*kid_count], &kids[*kid_count + 1]);
  split = __shfl_sync(0xffffffffu, split, 0);
  if (!split) return;
  *kid_count += 2;
  if (s.axis < 0) return;
  const Decision d = MakeDecision(nd, s);
  int nl = 0, nr = 0;
  const bool one = nd.end - nd.start <= 32;  // the warp holds them all: no second list
  for (int base = nd.start; base < nd.end; base += 32) {
    const int i = base + lane;
    const bool valid = i < nd.end;
    const int ref = valid ? idx[i] : 0;
    const bool left = valid && GoesLeft(d, box8, n_refs, ref);
    const unsigned lm = __ballot_sync(0xffffffffu, left), rm = __ballot_sync(0xffffffffu, valid && !left);
    const int at = left ? nd.start + nl + __popc(lm & lt) : d.mid + nr + __popc(rm & lt);
    if (valid) {
      if (left ? at < d.mid : at < nd.end) (one ? idx : tmp)[at] = ref;
      else atomicExch(&st->error, 6);
    }
    nl += __popc(lm);
    nr += __popc(rm);
  }
  if (one) return;
  __syncwarp();
  for (int i = nd.start + lane; i < nd.end; i += 32) idx[i] = tmp[i];
}

// One level of the small-node phase (nodes of more than kTinyRefs
// references). A round gives each warp one pending node, blocks first, so
// that few nodes lie on many SMs; its large nodes are taken by the whole
// block before. The children and the counts are kept by the warps and the
// block: one atomic per list and block instead of one per node on the same
// word.
__global__ void __launch_bounds__(kSmallWarps * 32, kSmallBlocks)
    SmallLevelKernel(const float4 *box8, int32_t *idx, int32_t *tmp, int n_refs, const PendingNode *in,
                     PendingNode *out, int q, int cap, PendingNode *tiny, int tiny_cap, int max_leaf,
                     BvhNode *sparse, int *used, uint8_t *last, SahStats *st) {
  __shared__ SmallShared sh;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int count = min(st->small_count[q], cap);
  // the list after next: its nodes were read by the level before this one
  if (blockIdx.x == 0 && threadIdx.x == 0) st->small_count[(q + 2) % 3] = 0;
  if (static_cast<int>(blockIdx.x) >= count) return;
  const KidLists lists = {{out, tiny}, {cap, tiny_cap}, {&st->small_count[(q + 1) % 3], &st->tiny_count}};
  if (threadIdx.x == 0) sh.leaves = sh.max_depth = sh.max_leaf = 0;
  NodeStats ns;  // lane 0's
  int kid_count = 0;
  for (int64_t base = blockIdx.x; base < count; base += static_cast<int64_t>(gridDim.x) * kSmallWarps) {
    const int64_t mine = base + static_cast<int64_t>(lane) * gridDim.x;
    bool large = false;
    if (lane < kSmallWarps && mine < count) large = in[mine].end - in[mine].start >= kTeamRefs;
    for (unsigned teams = __ballot_sync(0xffffffffu, large); teams; teams &= teams - 1) {
      const PendingNode nd = in[base + static_cast<int64_t>(__ffs(teams) - 1) * gridDim.x];
      if (!ValidNode(nd, n_refs) || nd.end - nd.start > kSmallRefs) {
        if (threadIdx.x == 0) atomicExch(&st->error, 7);
        continue;
      }
      if (wid == 0 && kid_count == kKids) {
        FlushKids(sh.kids[0], kid_count, lists, lane, st);
        kid_count = 0;
      }
      TeamNode(sh, nd, box8, idx, n_refs, max_leaf, sparse, used, last, &ns, &kid_count, st);
      __syncthreads();
    }
    const int64_t item = base + static_cast<int64_t>(wid) * gridDim.x;
    if (item >= count) continue;
    const PendingNode nd = in[item];
    const int n = nd.end - nd.start;
    if (n >= kTeamRefs) continue;
    if (!ValidNode(nd, n_refs) || n < 2) {
      if (lane == 0) atomicExch(&st->error, 7);
      continue;
    }
    if (kid_count == kKids) {
      FlushKids(sh.kids[wid], kid_count, lists, lane, st);
      kid_count = 0;
    }
    WarpNode(sh.bins[wid], sh.kids[wid], &kid_count, nd, box8, idx, tmp, n_refs, max_leaf, sparse, used, last, &ns,
             lane, st);
  }
  __syncthreads();
  const bool have = lane < kid_count;
  const int kind = have && sh.kids[wid][lane].end - sh.kids[wid][lane].start <= kTinyRefs ? 1 : 0;
  const unsigned kinds[2] = {__ballot_sync(0xffffffffu, have && !kind), __ballot_sync(0xffffffffu, kind)};
  if (lane < 2) sh.kid_count[lane][wid] = __popc(kinds[lane]);
  if (lane == 0) {
    if (ns.leaves) atomicAdd(&sh.leaves, ns.leaves);
    atomicMax(&sh.max_depth, ns.max_depth);
    atomicMax(&sh.max_leaf, ns.max_leaf);
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    int all = 0;
    for (int w = 0; w < kSmallWarps; ++w) all += sh.kid_count[threadIdx.x][w];
    sh.kid_base[threadIdx.x] = all ? atomicAdd(lists.count[threadIdx.x], all) : 0;
  }
  if (threadIdx.x == 32) {
    NodeStats b;
    b.leaves = sh.leaves, b.max_depth = sh.max_depth, b.max_leaf = sh.max_leaf;
    AddStats(b, st);
  }
  __syncthreads();
  if (have) {
    int at = sh.kid_base[kind] + __popc(kinds[kind] & ((1u << lane) - 1u));
    for (int w = 0; w < wid; ++w) at += sh.kid_count[kind][w];
    StoreKid(lists, sh.kids[wid][lane], kind, at, st);
  }
}

// Subtrees of at most kTinyRefs references, built to their leaves: a lane per
// reference, 32 / kTinyRefs subtrees per warp, all nodes of a subtree's level
// at once. A lane belongs to the node [s, e) of its group and evaluates the
// split after its own bin along each axis (the costs of empty bins repeat
// those of the occupied bin before, and the first bin at the minimum is
// taken), so no bins are needed: the boxes of both sides are unions over the
// group's lanes. Most nodes have this size: with a warp and its bins for
// each, the last levels took 60 us apiece; this kernel takes 35 us for all of
// them (87 k triangles).
__global__ void __launch_bounds__(kTinyWarps * 32) TinyKernel(const float4 *box8, int32_t *idx, int n_refs,
                                                              const PendingNode *roots, int cap, int max_leaf,
                                                              BvhNode *sparse, int *used, uint8_t *last,
                                                              SahStats *st) {
  constexpr int G = kTinyRefs;
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ int inverse[kTinyWarps][32];
  __shared__ int sh_leaves, sh_depth, sh_leaf;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int at = lane % G, g0 = lane - at;  // the lane's place in its group, the group's first lane
  const unsigned lt = (1u << lane) - 1u;
  const unsigned group = (G == 32 ? kAll : (1u << (G & 31)) - 1u) << g0;
  if (threadIdx.x == 0) sh_leaves = sh_depth = sh_leaf = 0;
  __syncthreads();
  const int count = min(st->tiny_count, cap);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kTinyWarps * (32 / G);
  NodeStats ns;
  for (int64_t base = (static_cast<int64_t>(blockIdx.x) * kTinyWarps + wid) * (32 / G); base < count; base += stride) {
    const int64_t item = base + lane / G;
    PendingNode nd{};
    bool open = item < count;
    if (open) {
      nd = roots[item];
      open = ValidNode(nd, n_refs) && nd.end - nd.start <= G;
      if (!open) atomicExch(&st->error, 7);
    }
    open = open && at < nd.end - nd.start;
    const int start = nd.start;
    int ref = open ? idx[start + at] : 0;
    const bool bad = open && static_cast<unsigned>(ref) >= static_cast<unsigned>(n_refs);
    if (bad) atomicExch(&st->error, 5);
    if (__ballot_sync(kAll, bad) & group) open = false;
    const bool mine = open;
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k) lo[k] = INFINITY, hi[k] = -INFINITY;
    if (open) LoadRef(box8, ref, lo, hi);
    int s = 0, e = open ? nd.end - start : 0;  // the lane's node, in the group
    while (__any_sync(kAll, open)) {
      const int n = e - s;
      float c[3];
      int bin[3];
      for (int k = 0; k < 3; ++k) {
        c[k] = Centroid(lo[k], hi[k]);
        bin[k] = BinOf(c[k], nd.clo[k], BinScale(nd.clo[k], nd.chi[k]));
      }
      // both sides' boxes of the lane's split along each axis
      float llo[3][3], lhi[3][3], rlo[3][3], rhi[3][3];
      int ln[3] = {0, 0, 0};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        for (int k = 0; k < 3; ++k)
          llo[a][k] = rlo[a][k] = INFINITY, lhi[a][k] = rhi[a][k] = -INFINITY;
      }
#pragma unroll 1
      for (int j = 0; j < G; ++j) {
        float olo[3], ohi[3];
        int ob[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          olo[k] = __shfl_sync(kAll, lo[k], g0 + j);
          ohi[k] = __shfl_sync(kAll, hi[k], g0 + j);
          ob[k] = __shfl_sync(kAll, bin[k], g0 + j);
        }
        if (j < s || j >= e) continue;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const bool left = ob[a] <= bin[a];
          ln[a] += left ? 1 : 0;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            if (left) llo[a][k] = fminf(llo[a][k], olo[k]), lhi[a][k] = fmaxf(lhi[a][k], ohi[k]);
            else rlo[a][k] = fminf(rlo[a][k], olo[k]), rhi[a][k] = fmaxf(rhi[a][k], ohi[k]);
          }
        }
      }
      float nlo[3], nhi[3];
      for (int k = 0; k < 3; ++k) nlo[k] = fminf(llo[0][k], rlo[0][k]), nhi[k] = fmaxf(lhi[0][k], rhi[0][k]);
      float cost = INFINITY;
      int key = 3 * kSahBins;  // axis and bin
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (!(__fsub_rn(nd.chi[a], nd.clo[a]) > 0.0f) || ln[a] >= n) continue;
        const float x = __fadd_rn(__fmul_rn(BoxArea(llo[a], lhi[a]), __int2float_rn(ln[a])),
                                  __fmul_rn(BoxArea(rlo[a], rhi[a]), __int2float_rn(n - ln[a])));
        if (x < cost) cost = x, key = a * kSahBins + bin[a];
      }
      // the node's cheapest: the lowest axis and bin at the lowest cost
      float best = INFINITY;
      int best_key = 3 * kSahBins;
#pragma unroll 1
      for (int j = 0; j < G; ++j) {
        const float oc = __shfl_sync(kAll, cost, g0 + j);
        const int ok = __shfl_sync(kAll, key, g0 + j);
        if (j >= s && j < e && (oc < best || (oc == best && ok < best_key))) best = oc, best_key = ok;
      }
      const int best_axis = best_key < 3 * kSahBins ? best_key / kSahBins : -1;
      const int axis = n == 1 ? -1 : DecideAxis(n, max_leaf, best_axis, best, nlo, nhi);
      const bool leaf = open && axis == -1, split = open && axis != -1;
      const int best_bin = best_key % kSahBins;
      const int my_bin = axis == 0 ? bin[0] : (axis == 1 ? bin[1] : bin[2]);
      const bool left = axis >= 0 ? my_bin <= best_bin : at - s < n / 2;
      const unsigned seg = n >= 32 ? kAll : ((1u << n) - 1u) << ((g0 + s) & 31);
      const unsigned lm = __ballot_sync(kAll, split && left) & seg;
      const int mid = s + __popc(lm), p = start + mid - 1;
      if (open && at == s) {
        ns.max_depth = max(ns.max_depth, nd.depth);
        WriteSlot(sparse, nd.parent, nlo, nhi, leaf ? ~(start + s) : p);
        if (leaf) {
          last[start + e - 1] = 1;
          ns.leaves += 1;
          ns.max_leaf = max(ns.max_leaf, n);
        } else {
          used[p] = 1;
        }
      }
      // a split node's references, left ones first, in order
      const int to = !split ? at : (left ? s + __popc(lm & lt) : mid + __popc(seg & ~lm & lt));
      inverse[wid][g0 + to] = lane;
      __syncwarp();
      const int from = inverse[wid][lane];
      __syncwarp();
      ref = __shfl_sync(kAll, ref, from);
      for (int k = 0; k < 3; ++k) {
        lo[k] = __shfl_sync(kAll, lo[k], from);
        hi[k] = __shfl_sync(kAll, hi[k], from);
        c[k] = __shfl_sync(kAll, c[k], from);
      }
      if (leaf) open = false;
      if (split) {
        nd.parent = 2 * p + (at < mid ? 0 : 1);
        nd.depth += 1;
        if (at < mid) e = mid;
        else s = mid;
      }
      // the children's centroid bounds (halves by position keep the node's)
      float clo[3], chi[3];
      for (int k = 0; k < 3; ++k) clo[k] = INFINITY, chi[k] = -INFINITY;
#pragma unroll 1
      for (int j = 0; j < G; ++j) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float oc = __shfl_sync(kAll, c[k], g0 + j);
          if (j >= s && j < e) clo[k] = fminf(clo[k], oc), chi[k] = fmaxf(chi[k], oc);
        }
      }
      if (split && axis >= 0) {
        for (int k = 0; k < 3; ++k) nd.clo[k] = clo[k], nd.chi[k] = chi[k];
      }
    }
    if (mine) idx[start + at] = ref;
  }
  atomicMax(&sh_depth, ns.max_depth);
  atomicMax(&sh_leaf, ns.max_leaf);
  if (ns.leaves) atomicAdd(&sh_leaves, ns.leaves);
  __syncthreads();
  if (threadIdx.x == 0) {
    NodeStats b;
    b.leaves = sh_leaves, b.max_depth = sh_depth, b.max_leaf = sh_leaf;
    AddStats(b, st);
  }
}

// Interior children per sparse entry (0 for positions that hold no node).
__global__ void ChildCountKernel(const BvhNode *sparse, const int *used, int n, int *kids) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n - 1) return;
  const BvhNode &nd = sparse[p];
  kids[p] = used[p] ? (nd.d.x >= 0 ? 1 : 0) + (nd.d.y >= 0 ? 1 : 0) : 0;
}

// Interior nodes into dense numbering: the root at 0, then the interior
// children of each node side by side (so one 128-byte line holds a pair of
// siblings), pairs in the order of their parents' split positions (`base`:
// exclusive scan of the child counts). Each node's thread writes its
// children; entry n - 1 of the sparse array is the root's virtual parent,
// whose slot 0 holds the root's box and link.
__global__ void DenseKernel(const BvhNode *sparse, const int *used, const int *base, int n, BvhNode *nodes) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const BvhNode &top = sparse[n - 1];
  const int root = top.d.x;
  if (root < 0) {
    // a single leaf: both slots hold it (as the host builder emits it)
    if (p == 0) {
      BvhNode nd{};
      nd.a = top.a;
      nd.b = top.a;
      nd.c = F4{top.c.x, top.c.y, top.c.x, top.c.y};
      nd.d = I4{root, root, 0, 0};
      nodes[0] = nd;
    }
    return;
  }
  auto renumbered = [&](int q) {
    BvhNode nd = sparse[q];
    int k = 0;
    if (nd.d.x >= 0) nd.d.x = 1 + base[q] + k++;
    if (nd.d.y >= 0) nd.d.y = 1 + base[q] + k++;
    nd.d.z = nd.d.w = 0;
    return nd;
  };
  if (p == 0) nodes[0] = renumbered(root);
  if (p >= n - 1 || !used[p]) return;
  const BvhNode &nd = sparse[p];
  int k = 0;
  if (nd.d.x >= 0) nodes[1 + base[p] + k++] = renumbered(nd.d.x);
  if (nd.d.y >= 0) nodes[1 + base[p] + k++] = renumbered(nd.d.y);
}

}  // namespace

namespace {

__global__ void CountKernel(const BvhNode *sparse, const int *kids, const int *base, int n, SahStats *st) {
  const int root = sparse[n - 1].d.x;
  st->root = root;
  st->nodes = root < 0 ? 1 : 1 + base[n - 2] + kids[n - 2];  // interior nodes
}

struct SahBuffers {
  float4 *box8 = nullptr;
  int32_t *tmp = nullptr;
  BvhNode *sparse = nullptr;
  int *used = nullptr, *rank = nullptr;
  PendingNode *level[2] = {nullptr, nullptr}, *small = nullptr, *small2 = nullptr, *tiny = nullptr;
  uint32_t *bins = nullptr;
  Decision *dec = nullptr;
  int2 *work = nullptr;
  int *chunk_left = nullptr, *first = nullptr;
  SahStats *st = nullptr;
  unsigned *cbounds = nullptr;
  void *scan_temp = nullptr;
  size_t scan_bytes = 0;
  int level_cap = 0, small_cap = 0, tiny_cap = 0, work_cap = 0;
};

// Places the buffers in `base` (nullptr: only sizes them); returns the bytes.
size_t Carve(int n, char *base, SahBuffers *b) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += (bytes + 255) / 256 * 256;
    return p;
  };
  const size_t m = static_cast<size_t>(std::max(n, 1));
  // level nodes are disjoint and hold >= kSmallRefs references each; small
  // nodes are disjoint and hold more than kTinyRefs; tiny ones are disjoint
  // and non-empty
  b->level_cap = n / kSmallRefs + 2;
  b->small_cap = n / (kTinyRefs + 1) + 2;
  b->tiny_cap = n + 1;
  b->work_cap = n / kMinChunk + b->level_cap + 1;
  b->box8 = reinterpret_cast<float4 *>(take(32 * m));
  b->tmp = reinterpret_cast<int32_t *>(take(4 * m));
  b->sparse = reinterpret_cast<BvhNode *>(take(sizeof(BvhNode) * m));
  b->used = reinterpret_cast<int *>(take(4 * m));
  b->rank = reinterpret_cast<int *>(take(4 * m));
  for (int k = 0; k < 2; ++k) b->level[k] = reinterpret_cast<PendingNode *>(take(sizeof(PendingNode) * b->level_cap));
  b->small = reinterpret_cast<PendingNode *>(take(sizeof(PendingNode) * b->small_cap));
  b->small2 = reinterpret_cast<PendingNode *>(take(sizeof(PendingNode) * b->small_cap));
  b->tiny = reinterpret_cast<PendingNode *>(take(sizeof(PendingNode) * b->tiny_cap));
  b->bins = reinterpret_cast<uint32_t *>(take(4ull * kNodeBinWords * b->level_cap));
  b->dec = reinterpret_cast<Decision *>(take(sizeof(Decision) * b->level_cap));
  b->work = reinterpret_cast<int2 *>(take(sizeof(int2) * b->work_cap));
  b->chunk_left = reinterpret_cast<int *>(take(4ull * b->work_cap));
  b->first = reinterpret_cast<int *>(take(4ull * (b->level_cap + 1)));
  b->st = reinterpret_cast<SahStats *>(take(sizeof(SahStats)));
  b->cbounds = reinterpret_cast<unsigned *>(take(6 * sizeof(unsigned)));
  b->scan_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, b->scan_bytes, static_cast<const int *>(nullptr), static_cast<int *>(nullptr),
                                std::max(n - 1, 1));
  b->scan_temp = take(b->scan_bytes);
  return off;
}

}  // namespace

size_t GpuSahScratchBytes(int n) {
  SahBuffers b;
  return Carve(n, nullptr, &b);
}

#define SAH_TRY(expr)                      \
  do {                                     \
    const cudaError_t _e = (expr);         \
    if (_e != cudaSuccess) return _e;      \
  } while (0)

cudaError_t BuildGpuSah(const float *boxes, int n, int max_leaf, void *scratch, BvhNode *nodes, int32_t *order,
                        uint8_t *last, GpuSahResult *res, cudaStream_t st) {
  *res = GpuSahResult{};
  if (n <= 0) return cudaSuccess;
  max_leaf = std::max(max_leaf, 1);
  SahBuffers b;
  Carve(n, static_cast<char *>(scratch), &b);
  int device = 0, sms = 1;
  SAH_TRY(cudaGetDevice(&device));
  SAH_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const unsigned init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
  SAH_TRY(cudaMemcpyAsync(b.cbounds, init, sizeof(init), cudaMemcpyHostToDevice, st));
  SAH_TRY(cudaMemsetAsync(b.st, 0, sizeof(SahStats), st));
  SAH_TRY(cudaMemsetAsync(last, 0, static_cast<size_t>(n), st));
  SAH_TRY(cudaMemsetAsync(b.used, 0, 4ull * n, st));
  SAH_TRY(cudaMemsetAsync(b.sparse, 0, sizeof(BvhNode) * static_cast<size_t>(n), st));
  PackKernel<<<Blocks(n, 256), 256, 0, st>>>(boxes, n, b.box8, order, b.cbounds);
  RootKernel<<<1, 1, 0, st>>>(n, b.cbounds, b.level[0], b.small, b.tiny, b.st);
  SAH_TRY(cudaGetLastError());
  SahStats h{};
  auto read_stats = [&]() {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, b.st, sizeof(h), cudaMemcpyDeviceToHost, st);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
  };
  // Levels are queued blindly; the lists' lengths are read back where they
  // can first have run out (a balanced tree's depth and some), then every few
  // levels. A level with nothing to do costs its launches.
  auto balanced = [](int64_t refs) {
    int d = 0;
    while ((1ll << d) < refs) ++d;
    return d;
  };
  const int chunk = ChunkRefs(n, sms);
  if (n >= kSmallRefs) {
    const int first_check = balanced(n / kSmallRefs) + 3;
    int cur = 0;
    for (int level = 0;; ++level) {
      if (level >= kMaxLevels || (level >= first_check && (level - first_check) % kLevelsPerCheck == 0)) {
        SAH_TRY(read_stats());
        if (h.error) {
          res->error = h.error;
          return cudaSuccess;
        }
        if (h.level_count[cur] == 0) break;
      }
      if (level >= kMaxLevels) {
        res->error = 1;
        return cudaSuccess;
      }
      const int nodes_max = static_cast<int>(std::min<int64_t>(b.level_cap, level < 31 ? 1ll << level : b.level_cap));
      const unsigned items_max = static_cast<unsigned>(std::min(b.work_cap, n / chunk + nodes_max));
      const unsigned init = Blocks(static_cast<int64_t>(nodes_max) * kNodeBinWords, 4 * kPlanThreads);
      LevelPlanKernel<<<1 + std::min(init, 2u * sms), kPlanThreads, 0, st>>>(b.level[cur], b.level_cap, cur, chunk,
                                                                             b.work_cap, b.work, b.first, b.bins,
                                                                             b.st);
      LevelBinKernel<<<items_max, kLevelThreads, 0, st>>>(b.box8, order, n, chunk, b.level[cur], b.work, b.bins, b.st);
      LevelSplitKernel<<<Blocks(static_cast<int64_t>(nodes_max) * 32, 128), 128, 0, st>>>(
          b.level[cur], cur, b.bins, max_leaf, b.dec, b.sparse, b.used, last, b.level[cur ^ 1], b.level_cap, b.small,
          b.small_cap, b.tiny, b.tiny_cap, b.st);
      LevelCountKernel<<<items_max, kLevelThreads, 0, st>>>(b.box8, order, n, chunk, b.level[cur], b.dec, b.work,
                                                            b.chunk_left, b.st);
      LevelScanKernel<<<nodes_max, kLevelThreads, 0, st>>>(b.dec, cur, b.level_cap, b.first, b.chunk_left, b.st);
      LevelScatterKernel<<<items_max, kLevelThreads, 0, st>>>(b.box8, order, n, chunk, b.tmp, b.level[cur], b.dec,
                                                              b.work, b.chunk_left, b.st);
      LevelCopyKernel<<<items_max, kLevelThreads, 0, st>>>(order, b.tmp, chunk, b.level[cur], b.dec, b.work, b.st);
      cur ^= 1;
    }
  }
  // the small-node phase, level by level
  if (n > kTinyRefs) {
    PendingNode *lists[2] = {b.small, b.small2};
    const unsigned grid = static_cast<unsigned>(sms) * kSmallBlocks;
    const int first_check = balanced(std::min(n, kSmallRefs) / kTinyRefs) + 4;
    for (int level = 0;; ++level) {
      const int q = level % 3;
      if (level >= kMaxSmallLevels || (level >= first_check && (level - first_check) % kLevelsPerCheck == 0)) {
        SAH_TRY(read_stats());
        if (h.error) {
          res->error = h.error;
          return cudaSuccess;
        }
        if (h.small_count[q] == 0) break;
      }
      if (level >= kMaxSmallLevels) {
        res->error = 1;
        return cudaSuccess;
      }
      SmallLevelKernel<<<grid, kSmallWarps * 32, 0, st>>>(b.box8, order, b.tmp, n, lists[level & 1],
                                                          lists[(level & 1) ^ 1], q, b.small_cap, b.tiny, b.tiny_cap,
                                                          max_leaf, b.sparse, b.used, last, b.st);
    }
  }
  TinyKernel<<<std::min(Blocks(n, kTinyWarps * 32), static_cast<unsigned>(sms) * 16u), kTinyWarps * 32, 0, st>>>(
      b.box8, order, n, b.tiny, b.tiny_cap, max_leaf, b.sparse, b.used, last, b.st);
  // b.tmp holds the child counts, b.rank their exclusive scan
  if (n >= 2) {
    ChildCountKernel<<<Blocks(n - 1, 256), 256, 0, st>>>(b.sparse, b.used, n, b.tmp);
    SAH_TRY(cub::DeviceScan::ExclusiveSum(b.scan_temp, b.scan_bytes, b.tmp, b.rank, n - 1, st));
  }
  DenseKernel<<<Blocks(std::max(n - 1, 1), 256), 256, 0, st>>>(b.sparse, b.used, b.rank, n, nodes);
  CountKernel<<<1, 1, 0, st>>>(b.sparse, b.tmp, b.rank, n, b.st);
  SAH_TRY(cudaGetLastError());
  SAH_TRY(cudaMemcpyAsync(&h, b.st, sizeof(h), cudaMemcpyDeviceToHost, st));
  SAH_TRY(cudaStreamSynchronize(st));
  res->error = h.error;
  res->nodes = h.nodes;
  res->leaves = static_cast<int64_t>(h.leaves);
  res->max_depth = h.max_depth;
  res->max_leaf = h.max_leaf;
  return cudaSuccess;
}

}  // namespace muon_gpu
