// kgpu_build.cu — the ImmutableKdTree soft construction on the device.
//
// The same tree, byte for byte, as the host builder (layout_build.cpp, the
// reference's construction.rs:413-539, 868-968, 1089-1175), built level by
// level instead of recursively.  A node of len points splits on axis level % K:
// its ideal pivot is ceil(len / 2) (soft_ideal_pivot with a power-of-two
// budget, clamped to [1, len]), v is the value at that place of the sorted
// coordinates, lt / le the number of values below / not above v, and
// update_pivot's nudge makes the pivot lt if lt > 0, else len if le == len
// (unsplittable, no stem), else le.  The stem is the value at the pivot and the
// left part is the points with a coordinate below it, so a split needs one
// order statistic and a partition by value, and no order inside the parts:
// leaves are sorted by source index at the end.
//
//  * Levels whose nodes are larger than a block's share (k_bracket, k_histogram,
//    k_find_bin, k_partition, k_select): the points lie in K coordinate columns
//    and an id column, every node's points side by side.  A sample brackets the
//    node's middle; a histogram of 1024 bins over the bracket (8192 on the first
//    levels) finds the bin that holds the ideal pivot; one pass moves the points
//    of lower bins to the front of the node, of higher bins to its end and the
//    bin's own into the gap, and a block per node then splits the gap (a
//    thousandth of the points) at the pivot's key.  Should a gap be too long for
//    a block (values spread over many exponents), the levels run once more with
//    such gaps bracketed and partitioned again, by all blocks (split_gaps).
//  * The last levels, once a node holds at most kShare points (k_finish): a
//    block per node sorts (node, key, place) words in registers once per level
//    and (leaf, source index, place) once more, and writes stems, leaf extents
//    and the rows of 3-D leaves.  Nodes that hold more than that (equal
//    coordinates move a pivot, and shares are full where n is just below a
//    power of two) are listed and split by the passes above for another level,
//    until their parts fit.
//
// What bounds it: the level passes are HBM streams of 4 (histogram) plus 2 x
// (4 K + 4) bytes per point and level in f32; k_finish is bound by instruction
// issue (seven sorting networks).  The stable radix
// sort per axis and prefix-sum partition of every axis's list on every level
// that this replaced moved about 117 bytes per point and level, over all 19
// levels of 16M points: 19.7 ms against 4.1 ms.
//
// One deliberate limit: a coordinate axis holding both -0.0 and +0.0 may give a
// stem of the other zero sign than the host builder's (which zero std's
// selection returns is unspecified; here that of the first zero in source
// order); every other input gives the host's bytes.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <limits>
#include <new>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/kiddo_gpu.h"
#include "kgpu_bitonic.cuh"
#include "kgpu_devbuf.h"
#include "kgpu_device.cuh"
#include "kgpu_internal.h"
#include "kgpu_launch.h"
#include "kgpu_tree_impl.h"

namespace kgpu {
namespace {

constexpr uint32_t kBucket = 32;

template <typename A>
__global__ void k_fill(A* __restrict__ p, uint64_t n, A v) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x)
    p[i] = v;
}

// ---- keys ----------------------------------------------------------------------
// Unsigned words that order like the coordinates; both zeros share a key.
template <typename A> struct OrdKey;
template <> struct OrdKey<float> {
  using U = uint32_t;
  __device__ __forceinline__ static U of(float x) {
    const uint32_t b = x == 0.f ? 0u : __float_as_uint(x);
    return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
  }
  __device__ __forceinline__ static float value(U k) {
    return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xffffffffu));
  }
  __device__ __forceinline__ static int bits(U w) { return 32 - __clz(int(w)); }
};
template <> struct OrdKey<double> {
  using U = unsigned long long;
  __device__ __forceinline__ static U of(double x) {
    const U b = x == 0.0 ? 0ull : static_cast<U>(__double_as_longlong(x));
    return b ^ ((b >> 63) ? ~0ull : 0x8000000000000000ull);
  }
  __device__ __forceinline__ static double value(U k) {
    return __longlong_as_double(
        static_cast<long long>(k ^ ((k >> 63) ? 0x8000000000000000ull : ~0ull)));
  }
  __device__ __forceinline__ static int bits(U w) { return 64 - __clzll((long long)w); }
};

// The points as K coordinate columns and their source indices.
template <typename A, int K>
struct Columns {
  A* c[K];
  uint32_t* id;
};

// Points of one block in k_finish: 64 leaves of a balanced tree.
constexpr uint32_t kShare = 2048;
constexpr uint32_t kShareLevels = 6;
// k_select: keys ranked by counting, and the bins of its histograms.
constexpr uint32_t kCandidates = 256;
constexpr int kGapBinsLog2 = 10;
constexpr uint32_t kGapBins = 1u << kGapBinsLog2;
constexpr uint64_t kTopNodes = 64;
// The longest gap of different keys that k_select's one block splits at once: a
// block reads about 40 GB/s, so this many points take 100 us or so.  Most gaps are
// a hundredth of it.
constexpr uint32_t kLongGap = 131072;
// Histogram bins by the level's nodes: enough that a node's gap is small beside
// it, few enough that a block's flush is small beside its points.
inline int bins_log2_of(uint64_t nodes) { return nodes <= kTopNodes ? 13 : nodes <= 8192 ? 10 : 6; }

// What one level knows of a node: its number on the level, its points
// [b, b + len), the bracket of its
// middle (keys [klo, khi] from a sample; vlo and inv spread the values in it
// over the inner bins), the bin of the ideal pivot, the points below and in it,
// and how many of each kind the partition has placed.
template <typename A>
struct alignas(16) Node {
  typename OrdKey<A>::U klo, khi;
  A vlo, inv;
  uint32_t index, b, len;
  uint32_t bin, below, in;
  uint32_t placed[3];
};

template <typename A>
__device__ __forceinline__ Node<A> new_node(uint32_t index, uint32_t b, uint32_t len) {
  Node<A> r;
  r.index = index;
  r.klo = r.khi = 0;
  r.vlo = r.inv = A(0);
  r.b = b;
  r.len = len;
  r.bin = r.below = r.in = 0;
  r.placed[0] = r.placed[1] = r.placed[2] = 0;
  return r;
}

__device__ __forceinline__ uint32_t ideal_pivot(uint32_t len) { return (len + 1) / 2; }

// The place whose key a node is split at: the ideal pivot, or `want` of it where the
// node is another's gap.  A place of len or more splits nothing.
__device__ __forceinline__ uint32_t wanted(const uint32_t* want, uint32_t node, uint32_t len) {
  return want ? want[node] : ideal_pivot(len);
}

// The bin of a coordinate: the first for keys below the bracket, the last for
// keys above it, and in between linear in the value (each operation is
// monotone, so bins order like keys).  GAP (a long gap's bracket): linear in the
// key instead, which resolves values over many exponents.
template <typename A, bool GAP>
__device__ __forceinline__ uint32_t bin_of(A x, typename OrdKey<A>::U klo,
                                           typename OrdKey<A>::U khi, A vlo, A inv,
                                           uint32_t bins) {
  const auto k = OrdKey<A>::of(x);
  if (k < klo) return 0;
  if (k > khi) return bins - 1;
  if constexpr (GAP) {
    // half of the bins or fewer, so that the last inner bin is never passed
    const int shift = OrdKey<A>::bits(khi - klo) - (30 - __clz(int(bins)));
    return 1u + uint32_t((k - klo) >> (shift > 0 ? shift : 0));
  }
  return 1u + (inv > A(0) ? min(uint32_t(mul_rn(sub_rn(x, vlo), inv)), bins - 3) : 0u);
}

template <typename A, int K>
__global__ void k_columns(const A* __restrict__ pts, uint64_t n, Columns<A, K> out) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
#pragma unroll
    for (int d = 0; d < K; ++d) out.c[d][i] = pts[i * K + d];
    out.id[i] = uint32_t(i);
  }
}

template <typename A>
__global__ void k_root(Node<A>* __restrict__ nodes, uint32_t n) {
  nodes[0] = new_node<A>(0, 0, n);
}

// The last node that begins at or before position p: the one holding p if any
// does, as empty nodes begin where the next one does.
template <typename A>
__device__ __forceinline__ uint32_t node_at(const Node<A>* nodes, uint32_t count, uint32_t p) {
  uint32_t lo = 0, hi = count;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (nodes[mid].b <= p) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Calls f(node, first, last) for the piece of every node inside the block's
// share of the positions (`share` per block, in order); the nodes need not cover
// them.  Uniform in the block.
template <typename A, typename F>
__device__ __forceinline__ void for_each_piece(const Node<A>* nodes, uint32_t count, uint32_t n,
                                               uint32_t share, F&& f) {
  const uint64_t first = uint64_t(blockIdx.x) * share;
  if (first >= n) return;
  const uint32_t p0 = uint32_t(first);
  const uint32_t end = uint32_t(first + share < n ? first + share : n);
  uint32_t node = node_at(nodes, count, p0), stop;
  do {
    const uint32_t b = nodes[node].b;
    stop = b + nodes[node].len;
    const uint32_t p = max(p0, b), last = min(end, stop);
    if (last > p) f(node, p, last);
    ++node;
  } while (stop < end && node < count);
}

// Minimum and maximum over the block (uniform result).
template <typename U>
__device__ __forceinline__ void block_min_max(U& lo, U& hi, U* red) {
  for (int o = 16; o > 0; o >>= 1) {
    const U a = __shfl_xor_sync(FULL, lo, o), b = __shfl_xor_sync(FULL, hi, o);
    lo = a < lo ? a : lo;
    hi = b > hi ? b : hi;
  }
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    red[warp] = lo;
    red[32 + warp] = hi;
  }
  __syncthreads();
  for (int w = 0; w < warps; ++w) {
    lo = red[w] < lo ? red[w] : lo;
    hi = red[32 + w] > hi ? red[32 + w] : hi;
  }
  __syncthreads();
}

// Place i of a sample of 256 among len points: anywhere in the i-th of 256 equal
// shares, by a multiplicative hash of the place
// and the node.  Evenly spaced places met the period of ordered inputs: in a
// raster whose rows divide the spacing every sample has the same coordinate, the
// bracket misses the middle and one block sorts out the whole node (256^3 grid,
// x fastest: 84 ms, 4.3 now; 2048 x 2048 image 13.5 ms, 1.2 now).
__device__ __forceinline__ uint32_t sample_place(uint32_t i, uint32_t b, uint32_t len) {
  constexpr uint32_t kPhi = 0x9e3779b9u;  // 2^32 over the golden ratio (Knuth)
  uint32_t h = (i + kPhi * (b ^ (len << 1))) * kPhi;
  h = (h ^ (h >> 15)) * kPhi;
  h = (h ^ (h >> 13)) * kPhi;
  h ^= h >> 16;
  return uint32_t((uint64_t(i) * len + ((uint64_t(h) * len) >> 32)) >> 8);
}

// The bracket of every node's middle (of its wanted place, in general), a block per
// node: 256 points spread over the node (sample_place), ranked by counting; the
// bracket runs five standard deviations (8) of the sample's median to either side,
// about a third of the points.  A middle outside it only makes k_select work longer (203 us once in
// 13 levels of 16M points at four deviations, against 5 to 14).  Quantiles hold
// for any spread of the values: over the node's whole range, bins linear in the
// key put 1/64 of the points in one bin where the range holds zero (all
// exponents; k_select then took 3.8 of 8.1 ms), and bins linear in the value put
// them all in one beside an outlier.  1024 samples took 34 us a level for 6.
template <typename A>
__global__ void __launch_bounds__(256) k_bracket(const A* __restrict__ col,
                                                  Node<A>* __restrict__ nodes, uint32_t count,
                                                  uint32_t bins,
                                                  const uint32_t* __restrict__ want) {
  using U = typename OrdKey<A>::U;
  constexpr uint32_t nt = 256, half = 40;  // sample_place shares by nt
  __shared__ U key[nt];
  __shared__ U ends[2];
  const uint32_t tid = threadIdx.x;
  for (uint32_t node = blockIdx.x; node < count; node += gridDim.x) {
    const uint32_t b = nodes[node].b, len = nodes[node].len;
    if (len > 1) {
      const U k = OrdKey<A>::of(col[b + sample_place(tid, b, len)]);
      key[tid] = k;
      __syncthreads();
      uint32_t rank = 0;
#pragma unroll 8
      for (uint32_t i = 0; i < nt; ++i) rank += key[i] < k || (key[i] == k && i < tid) ? 1u : 0u;
      const uint32_t mid = want ? uint32_t(uint64_t(want[node]) * nt / len) : nt / 2;
      if (rank == (mid > half ? mid - half : 0u)) ends[0] = k;
      if (rank == min(mid + half, nt - 1)) ends[1] = k;
      __syncthreads();
      if (tid == 0) {
        const A lo = OrdKey<A>::value(ends[0]), hi = OrdKey<A>::value(ends[1]);
        const A w = sub_rn(hi, lo);
        nodes[node].klo = ends[0];
        nodes[node].khi = ends[1];
        nodes[node].vlo = lo;
        // finite and positive, or every point of the bracket shares a bin
        const A inv = A(bins - 2) / w;
        nodes[node].inv = w > A(0) && w < inf_of<A>() && inv < inf_of<A>() ? inv : A(0);
      }
      __syncthreads();
    }
  }
}

// hist[node][bin]: the node's points by the bin of their key.  16M f32 points:
// 46 us a level, bound by the shared-memory atomics of the inner bins (80 us
// with one load in flight per thread).
template <typename A, bool GAP = false>
__global__ void __launch_bounds__(256) k_histogram(
    const A* __restrict__ col, const Node<A>* __restrict__ nodes, uint32_t count, uint32_t n,
    uint32_t share, int bins_log2, uint32_t* __restrict__ hist) {
  extern __shared__ uint32_t sh[];
  const uint32_t bins = 1u << bins_log2;
  for_each_piece(nodes, count, n, share, [&](uint32_t node, uint32_t p, uint32_t last) {
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    const auto klo = nodes[node].klo, khi = nodes[node].khi;
    const A vlo = nodes[node].vlo, inv = nodes[node].inv;
    // the two outer bins hold most points: counted in registers
    uint32_t first = 0, final = 0;
    for (uint32_t r = p; r < last; r += 256 * 8) {
      A x[8];  // eight loads in flight
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t i = r + j * 256 + threadIdx.x;
        x[j] = i < last ? col[i] : A(0);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (r + j * 256 + threadIdx.x >= last) continue;
        const uint32_t at = bin_of<A, GAP>(x[j], klo, khi, vlo, inv, bins);
        if (at == 0) ++first;
        else if (at == bins - 1) ++final;
        else atomicAdd(sh + at, 1u);
      }
    }
    first = __reduce_add_sync(FULL, first);
    final = __reduce_add_sync(FULL, final);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(sh, first);
      atomicAdd(sh + bins - 1, final);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x)
      if (sh[i]) atomicAdd(hist + uint64_t(node) * bins + i, sh[i]);
    __syncthreads();
  });
}

// The bin of counts[0..bins) that holds place `at` (at < their sum), the
// entries before it and in it: one block, `bins` a multiple of its threads or
// fewer (the other threads hold nothing).  `scan` holds a word per warp and
// the three results.
__device__ __forceinline__ void block_find_bin(const uint32_t* counts, uint32_t bins, uint32_t at,
                                               uint32_t* scan, uint32_t& bin, uint32_t& below,
                                               uint32_t& in) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, warps = blockDim.x >> 5;
  const uint32_t per = bins > blockDim.x ? bins / blockDim.x : 1;
  uint32_t sum = 0;
  if (tid * per < bins)
    for (uint32_t i = 0; i < per; ++i) sum += counts[tid * per + i];
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(FULL, incl, o);
    if (lane >= uint32_t(o)) incl += v;
  }
  __syncthreads();
  if (lane == 31) scan[tid >> 5] = incl;
  __syncthreads();
  uint32_t run = incl - sum;
  for (uint32_t w = 0; w < (tid >> 5); ++w) run += scan[w];
  if (run <= at && at - run < sum) {  // one thread
    uint32_t i = tid * per;
    while (at - run >= counts[i]) run += counts[i++];
    scan[warps] = i;
    scan[warps + 1] = run;
    scan[warps + 2] = counts[i];
  }
  __syncthreads();
  bin = scan[warps];
  below = scan[warps + 1];
  in = scan[warps + 2];
}

// One block per node.  A node whose ideal pivot is its length (0 or 1 points)
// has nothing to split: all of it is its gap.
template <typename A>
__global__ void __launch_bounds__(256) k_find_bin(Node<A>* __restrict__ nodes, uint32_t count,
                                                  const uint32_t* __restrict__ hist,
                                                  uint32_t bins,
                                                  const uint32_t* __restrict__ want) {
  __shared__ uint32_t scan[16];
  for (uint32_t node = blockIdx.x; node < count; node += gridDim.x) {
    const uint32_t len = nodes[node].len, at = wanted(want, node, len);
    uint32_t bin = 0, below = 0, in = len;
    if (at < len) block_find_bin(hist + uint64_t(node) * bins, bins, at, scan, bin, below, in);
    if (threadIdx.x == 0) {
      nodes[node].bin = bin;
      nodes[node].below = below;
      nodes[node].in = in;
    }
    __syncthreads();
  }
}

// Moves every node's points from `in` to `out`: those of bins below the
// pivot's first, then the pivot's bin, then the rest.  2048 points at a time: a
// thread holds 8, counts its warp's by kind with ballots, and one thread takes
// the block's room from the node's counters, so each kind is written as one run
// per block and round.  16M f32 points: 113 us a level (4.5 TB/s), 145 with each
// load next to its ballot.
template <typename A, int K, bool GAP = false>
__global__ void __launch_bounds__(256) k_partition(
    Columns<A, K> in, Columns<A, K> out, const A* __restrict__ col,
    Node<A>* __restrict__ nodes, uint32_t count, uint32_t n, uint32_t share, int bins_log2) {
  constexpr int kItems = 8;
  __shared__ uint32_t warp_n[8][3], base[3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for_each_piece(nodes, count, n, share, [&](uint32_t node, uint32_t p, uint32_t last) {
    const uint32_t b = nodes[node].b, below = nodes[node].below, inside = nodes[node].in;
    const uint32_t bin = nodes[node].bin;
    // (only long gaps have points where they are nodes)
    const bool split = GAP || ideal_pivot(nodes[node].len) < nodes[node].len;
    const auto klo = nodes[node].klo, khi = nodes[node].khi;
    const A vlo = nodes[node].vlo, inv = nodes[node].inv;
    for (uint32_t r = p; r < last; r += 256 * kItems) {
      A c[kItems][K];
      uint32_t id[kItems], kinds = 0;  // two bits per item; 3: no point
      uint32_t cnt[3] = {0, 0, 0};
      uint32_t rank[kItems];
      // every load before the first ballot, so all are in flight together; the
      // split axis is read again (an L1 hit), as selecting it from c[j] by its
      // number would put c in local memory
      A x[kItems];
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const uint32_t i = r + (warp * kItems + j) * 32 + lane;
        if (i < last) {
          x[j] = col[i];
#pragma unroll
          for (int a = 0; a < K; ++a) c[j][a] = in.c[a][i];
          id[j] = in.id[i];
        }
      }
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const uint32_t i = r + (warp * kItems + j) * 32 + lane;
        uint32_t kind = 3;
        if (i < last) {
          const uint32_t bi = bin_of<A, GAP>(x[j], klo, khi, vlo, inv, 1u << bins_log2);
          kind = !split || bi == bin ? 1 : (bi < bin ? 0 : 2);
        }
        kinds |= kind << (2 * j);
        const unsigned below_me = (1u << lane) - 1u;
#pragma unroll
        for (uint32_t k = 0; k < 3; ++k) {
          const unsigned m = __ballot_sync(FULL, kind == k);
          if (kind == k) rank[j] = cnt[k] + __popc(m & below_me);
          cnt[k] += __popc(m);
        }
      }
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) warp_n[warp][k] = cnt[k];
      }
      __syncthreads();
      if (threadIdx.x < 3) {
        uint32_t run = 0;
        for (int w = 0; w < 8; ++w) {
          const uint32_t v = warp_n[w][threadIdx.x];
          warp_n[w][threadIdx.x] = run;
          run += v;
        }
        base[threadIdx.x] = run ? atomicAdd(&nodes[node].placed[threadIdx.x], run) : 0u;
      }
      __syncthreads();
      const uint32_t at0 = b + base[0] + warp_n[warp][0];
      const uint32_t at1 = b + below + base[1] + warp_n[warp][1];
      const uint32_t at2 = b + below + inside + base[2] + warp_n[warp][2];
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const uint32_t kind = (kinds >> (2 * j)) & 3u;
        if (kind != 3) {
          const uint32_t o = (kind == 0 ? at0 : kind == 1 ? at1 : at2) + rank[j];
#pragma unroll
          for (int a = 0; a < K; ++a) out.c[a][o] = c[j][a];
          out.id[o] = id[j];
        }
      }
      __syncthreads();
    }
  });
}

// Whether a node's gap holds one key only, its klo: the bin of a bracket of one key.
template <typename A>
__device__ __forceinline__ bool one_key(const Node<A>& node) {
  return node.bin == 1 && node.klo == node.khi;
}

// ---- long gaps ---------------------------------------------------------------
// The gaps above kLongGap as nodes of their own (the other nodes are left empty)
// with the place wanted in each; *any tells whether there are such.
template <typename A>
__global__ void k_list_gaps(const Node<A>* __restrict__ nodes, uint32_t count,
                            Node<A>* __restrict__ gaps, uint32_t* __restrict__ want,
                            uint32_t* __restrict__ any) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const Node<A> nd = nodes[i];
    const uint32_t ideal = ideal_pivot(nd.len);
    const bool is_long = ideal < nd.len && nd.in > kLongGap && !one_key(nd);
    gaps[i] = new_node<A>(nd.index, is_long ? nd.b + nd.below : nd.b, is_long ? nd.in : 0u);
    want[i] = is_long ? ideal - nd.below : 0u;
    if (is_long) *any = 1;
  }
}
// Their partition becomes the nodes'.
template <typename A>
__global__ void k_take_gaps(Node<A>* __restrict__ nodes, uint32_t count,
                            const Node<A>* __restrict__ gaps) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    if (!gaps[i].len) continue;
    nodes[i].below += gaps[i].below;
    nodes[i].in = gaps[i].in;
    nodes[i].bin = gaps[i].bin;
    nodes[i].klo = gaps[i].klo;
    nodes[i].khi = gaps[i].khi;
  }
}
template <typename A, int K>
__global__ void __launch_bounds__(256) k_copy_gaps(Columns<A, K> in, Columns<A, K> out,
                                                   const Node<A>* __restrict__ gaps,
                                                   uint32_t count, uint32_t n, uint32_t share) {
  for_each_piece(gaps, count, n, share, [&](uint32_t, uint32_t p, uint32_t last) {
    for (uint32_t i = p + threadIdx.x; i < last; i += blockDim.x) {
#pragma unroll
      for (int a = 0; a < K; ++a) out.c[a][i] = in.c[a][i];
      out.id[i] = in.id[i];
    }
  });
}

// The sign of a zero stem: that of the node's first zero in source order.
// Points [first, last) of the column; block-wide, uniform result.
template <typename A, int K>
__device__ A zero_stem(const Columns<A, K>& cur, int d, uint32_t first, uint32_t last,
                       uint32_t* best) {
  __syncthreads();
  if (threadIdx.x == 0) *best = 0xffffffffu;
  __syncthreads();
  const A* col = cur.c[d];
  for (uint32_t i = first + threadIdx.x; i < last; i += blockDim.x)
    if (col[i] == A(0)) atomicMin(best, cur.id[i]);
  __syncthreads();
  const uint32_t id = *best;
  __shared__ A found;
  for (uint32_t i = first + threadIdx.x; i < last; i += blockDim.x)
    if (cur.id[i] == id) found = col[i];
  __syncthreads();
  const A r = found;
  __syncthreads();
  return r;
}

// Finds the key at a node's ideal pivot among the gap (the points of its bin), moves
// the gap's points below it to the front and above it to the back, sets the stem
// and returns the pivot (the node's length: no split), by the whole block.  The key is found by
// histograms of ever narrower ranges until at most kCandidates points are in
// range, whose keys are ranked by counting; the points move once, a thread
// holding one each, or through `tmp` (the other set of columns, free now) when
// the gap has more points than the block threads.  A gap of one key stays as it
// is.  Where `too_long` is given, a gap above kLongGap of different keys sets it
// and its node is left whole (and so are others, once it is set): the caller
// starts again.
template <typename A, int K>
__device__ __forceinline__ uint32_t split_node(const Columns<A, K>& cur, const Columns<A, K>& tmp,
                                               int d, const Node<A>& nd, A* __restrict__ stems,
                                               uint32_t* __restrict__ too_long) {
  using U = typename OrdKey<A>::U;
  __shared__ U key[kCandidates];
  __shared__ uint32_t bins[kGapBins], scan[40];
  __shared__ U red[64], found_key;
  __shared__ uint32_t found[2], placed[3], zero_id, give_up;
  const uint32_t tid = threadIdx.x, nt = blockDim.x;
  const uint32_t b = nd.b, len = nd.len, ideal = ideal_pivot(len);
  if (ideal >= len) return len;
  const uint32_t lo = nd.below, cnt = nd.in;
  const A* gap = cur.c[d] + b + lo;
  // r: the wanted place among the `in` points of keys [kmin, kmax]
  uint32_t r = ideal - lo, in = cnt, before = 0;
  U kmin = 0, kmax = ~U(0);
  if (one_key(nd)) {
    kmin = kmax = nd.klo;
  } else if (cnt > kCandidates) {
    const bool check = too_long && cnt > kLongGap;
    if (check) {
      if (tid == 0) give_up = atomicAdd(too_long, 0u);
      __syncthreads();
      if (give_up) return len;
    }
    kmin = ~U(0);
    kmax = 0;
#pragma unroll 4
    for (uint32_t i = tid; i < cnt; i += nt) {
      const U k = OrdKey<A>::of(gap[i]);
      kmin = k < kmin ? k : kmin;
      kmax = k > kmax ? k : kmax;
    }
    block_min_max(kmin, kmax, red);
    if (check && kmin != kmax) {
      if (tid == 0) *too_long = 1;
      return len;
    }
  }
  const bool moves = kmin != kmax;
  while (in > kCandidates && kmin != kmax) {
    const int width = OrdKey<A>::bits(kmax - kmin);
    const int shift = width > kGapBinsLog2 ? width - kGapBinsLog2 : 0;
    for (uint32_t i = tid; i < kGapBins; i += nt) bins[i] = 0;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = tid; i < cnt; i += nt) {
      const U k = OrdKey<A>::of(gap[i]);
      if (k >= kmin && k <= kmax) atomicAdd(bins + uint32_t((k - kmin) >> shift), 1u);
    }
    __syncthreads();
    uint32_t bin, below;
    block_find_bin(bins, kGapBins, r, scan, bin, below, in);
    __syncthreads();
    before += below;
    r -= below;
    kmin += U(bin) << shift;
    const U top = kmin + ((U(1) << shift) - 1);
    kmax = top < kmax && top >= kmin ? top : kmax;
  }
  U v = kmin;
  uint32_t lt = lo + before, equals = in;  // points below v, points equal to v
  if (kmin != kmax) {
    // rank the candidates by counting
    if (tid == 0) placed[0] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < cnt; i += nt) {
      const U k = OrdKey<A>::of(gap[i]);
      if (k >= kmin && k <= kmax) key[atomicAdd(placed, 1u)] = k;
    }
    __syncthreads();
    if (tid < in) {
      const U k = key[tid];
      uint32_t less = 0, same = 0;
      for (uint32_t i = 0; i < in; ++i) {
        less += key[i] < k ? 1u : 0u;
        same += key[i] == k ? 1u : 0u;
      }
      if (less <= r && r - less < same) {  // every holder writes the same
        found_key = k;
        found[0] = less;
        found[1] = same;
      }
    }
    __syncthreads();
    v = found_key;
    lt = lo + before + found[0];
    equals = found[1];
  }
  const uint32_t le = lt + equals;
  // below v, v, above v
  if (tid < 3) placed[tid] = 0;
  __syncthreads();
  const uint32_t start1 = lt - lo, start2 = le - lo;
  if (!moves) {
    // all of the gap is v
  } else if (cnt <= nt) {
    A c[K];
    uint32_t id = 0, o = 0;
    if (tid < cnt) {
      const U k = OrdKey<A>::of(gap[tid]);
      const int kind = k < v ? 0 : k == v ? 1 : 2;
      o = (kind == 0 ? 0u : kind == 1 ? start1 : start2) + atomicAdd(placed + kind, 1u);
#pragma unroll
      for (int a = 0; a < K; ++a) c[a] = cur.c[a][b + lo + tid];
      id = cur.id[b + lo + tid];
    }
    __syncthreads();
    if (tid < cnt) {
#pragma unroll
      for (int a = 0; a < K; ++a) cur.c[a][b + lo + o] = c[a];
      cur.id[b + lo + o] = id;
    }
  } else {
    const unsigned below_me = (1u << (tid & 31)) - 1u;
    for (uint32_t i0 = 0; i0 < cnt; i0 += nt) {
      const uint32_t i = i0 + tid;
      int kind = 3;
      if (i < cnt) {
        const U k = OrdKey<A>::of(gap[i]);
        kind = k < v ? 0 : k == v ? 1 : 2;
      }
      uint32_t o = 0;
#pragma unroll
      for (int j = 0; j < 3; ++j) {  // one atomic per warp and kind
        const unsigned m = __ballot_sync(FULL, kind == j);
        if (kind == j) {
          const int lead = __ffs(m) - 1;
          uint32_t at = 0;
          if (int(tid & 31) == lead) at = atomicAdd(placed + j, uint32_t(__popc(m)));
          at = __shfl_sync(m, at, lead);
          o = b + lo + (j == 0 ? 0u : j == 1 ? start1 : start2) + at + __popc(m & below_me);
        }
      }
      if (kind != 3) {
        const uint32_t s = b + lo + i;
#pragma unroll
        for (int a = 0; a < K; ++a) tmp.c[a][o] = cur.c[a][s];
        tmp.id[o] = cur.id[s];
      }
    }
    __syncthreads();
    for (uint32_t i = tid; i < cnt; i += nt) {
      const uint32_t s = b + lo + i;
#pragma unroll
      for (int a = 0; a < K; ++a) cur.c[a][s] = tmp.c[a][s];
      cur.id[s] = tmp.id[s];
    }
  }
  __syncthreads();
  const A value = OrdKey<A>::value(v);
  if (value != value) return len;  // a NaN at the ideal pivot splits nothing
  const uint32_t pivot = lt > 0 ? lt : (le >= len ? len : le);
  if (pivot == len) return len;
  U k = v;
  if (pivot != lt) {  // the smallest key above v
    U least = ~U(0), most = 0;
    for (uint32_t i = b + le + tid; i < b + len; i += nt) {
      const U kk = OrdKey<A>::of(cur.c[d][i]);
      least = kk < least ? kk : least;
    }
    block_min_max(least, most, red);
    k = least;
  }
  A stem = OrdKey<A>::value(k);
  if (stem == A(0)) stem = zero_stem(cur, d, b + pivot, b + len, &zero_id);
  if (tid == 0) stems[nd.index] = stem;
  return pivot;
}

// One block per node: its split and its two children.
template <typename A, int K>
__global__ void __launch_bounds__(1024, 2) k_select(
    Columns<A, K> cur, Columns<A, K> tmp, int d,
    const Node<A>* __restrict__ nodes, uint32_t count,
    A* __restrict__ stems, Node<A>* __restrict__ next, uint32_t* __restrict__ too_long) {
  for (uint32_t node = blockIdx.x; node < count; node += gridDim.x) {
    const uint32_t pivot = split_node(cur, tmp, d, nodes[node], stems, too_long);
    if (threadIdx.x < 2) {
      const uint32_t b = nodes[node].b, len = nodes[node].len;
      const uint32_t child = 2 * nodes[node].index + threadIdx.x;
      next[2 * uint64_t(node) + threadIdx.x] =
          threadIdx.x ? new_node<A>(child, b + pivot, len - pivot) : new_node<A>(child, b, pivot);
    }
    __syncthreads();
  }
}

// ---- the last levels --------------------------------------------------------------
// (node, key, place) and (leaf, source index, place) as one sortable word.
template <typename A> struct PlaceKey;
template <> struct PlaceKey<float> {
  unsigned long long v;  // 20 bits node (below 64), 32 key, 12 place
  __device__ __forceinline__ static PlaceKey make(uint32_t node, uint32_t key, uint32_t place) {
    return {(static_cast<unsigned long long>(node) << 44) |
            (static_cast<unsigned long long>(key) << 12) | place};
  }
  __device__ __forceinline__ static PlaceKey last() { return {kLastWord}; }
  __device__ __forceinline__ bool operator<(const PlaceKey& o) const { return word_less(v, o.v); }
  __device__ __forceinline__ uint32_t node() const { return uint32_t(v >> 44); }
  __device__ __forceinline__ uint32_t key() const { return uint32_t(v >> 12); }
  __device__ __forceinline__ uint32_t place() const { return uint32_t(v) & 0xfffu; }
  __device__ __forceinline__ PlaceKey from_lane(int mask) const {
    return {__shfl_xor_sync(FULL, v, mask)};
  }
};
template <> struct PlaceKey<double> {
  unsigned long long k;
  uint32_t p;  // 16 bits node, 16 place
  __device__ __forceinline__ static PlaceKey make(uint32_t node, unsigned long long key,
                                                  uint32_t place) {
    return {key, (node << 16) | place};
  }
  __device__ __forceinline__ static PlaceKey last() { return {~0ull, ~0u}; }
  __device__ __forceinline__ bool operator<(const PlaceKey& o) const {
    const uint32_t a = p >> 16, b = o.p >> 16;
    return a != b ? a < b : (k < o.k || (k == o.k && p < o.p));
  }
  __device__ __forceinline__ uint32_t node() const { return p >> 16; }
  __device__ __forceinline__ unsigned long long key() const { return k; }
  __device__ __forceinline__ uint32_t place() const { return p & 0xffffu; }
  __device__ __forceinline__ PlaceKey from_lane(int mask) const {
    return {__shfl_xor_sync(FULL, k, mask), __shfl_xor_sync(FULL, p, mask)};
  }
};
}  // namespace
// in shared memory, one pad slot after every 16
template <>
struct KeyStore<PlaceKey<float>> {
  unsigned long long* v;
  __host__ __device__ static constexpr size_t bytes(uint32_t n) { return (n + n / 16) * 8; }
  __device__ static KeyStore at(unsigned char* p, uint32_t) {
    return {reinterpret_cast<unsigned long long*>(p)};
  }
  __device__ __forceinline__ PlaceKey<float> get(uint32_t i) const { return {v[i + (i >> 4)]}; }
  __device__ __forceinline__ void put(uint32_t i, const PlaceKey<float>& k) { v[i + (i >> 4)] = k.v; }
};
template <>
struct KeyStore<PlaceKey<double>> {
  unsigned long long* v;
  uint32_t* p;
  __host__ __device__ static constexpr size_t bytes(uint32_t n) { return (n + n / 16) * 12; }
  __device__ static KeyStore at(unsigned char* m, uint32_t n) {
    unsigned long long* v = reinterpret_cast<unsigned long long*>(m);
    return {v, reinterpret_cast<uint32_t*>(v + n + n / 16)};
  }
  __device__ __forceinline__ PlaceKey<double> get(uint32_t i) const {
    return {v[i + (i >> 4)], p[i + (i >> 4)]};
  }
  __device__ __forceinline__ void put(uint32_t i, const PlaceKey<double>& k) {
    v[i + (i >> 4)] = k.k;
    p[i + (i >> 4)] = k.p;
  }
};
namespace {

template <typename A, int K>
constexpr size_t finish_smem() {
  return KeyStore<PlaceKey<A>>::bytes(kShare) + size_t(K) * kShare * sizeof(A) + kShare * 4;
}

template <typename A>
__device__ __forceinline__ void put_row(uint8_t* rows, uint32_t p, A x, A y, A z, uint32_t it);

// One block of 256 threads per node of level `level`, 8 keys per thread: the
// remaining `levels` levels and the leaf order, all in registers and shared
// memory.  Writes the stems, each leaf's begin and length and, in leaf order,
// the rows of 3-D leaves (arena != null) or the source indices.  A node above
// kShare points is only counted in *too_big.
//
// A part of sub-level j has a slot of kShare >> j positions while every part
// fits its slot (the parts of a split are equal but for equal coordinates), so
// the networks only sort runs of that length: 266 steps in all for seven sorts
// against 462 for whole-block ones.  Once some part does not fit, the parts lie
// side by side (`dense`) and the whole block is sorted on (part, key).
template <typename A, int K>
__global__ void __launch_bounds__(256, sizeof(A) == 4 ? 4 : 2) k_finish(
    Columns<A, K> cur, const Node<A>* __restrict__ nodes, uint32_t level,
    uint32_t levels, A* __restrict__ stems, const uint32_t* __restrict__ items,
    uint8_t* __restrict__ arena, uint32_t* __restrict__ ids, uint32_t* __restrict__ leaf_b,
    uint32_t* __restrict__ leaf_len, uint32_t* __restrict__ too_big) {
  constexpr int T = 256, E = kShare / T;
  constexpr uint32_t kNone = 0xffffffffu;
  using Key = PlaceKey<A>;
  extern __shared__ __align__(16) unsigned char smem[];
  KeyStore<Key> ks = KeyStore<Key>::at(smem, kShare);
  A* cs = reinterpret_cast<A*>(smem + KeyStore<Key>::bytes(kShare));  // [K][kShare]
  uint32_t* sid = reinterpret_cast<uint32_t*>(cs + size_t(K) * kShare);
  __shared__ uint32_t begin[2][65];
  __shared__ int overflow;
  const uint32_t tid = threadIdx.x, node = nodes[blockIdx.x].index;
  const uint32_t b0 = nodes[blockIdx.x].b, len = nodes[blockIdx.x].len;
  if (len > kShare) {
    if (tid == 0) atomicAdd(too_big, 1u);
    return;
  }
  for (uint32_t i = tid; i < len; i += T) {
#pragma unroll
    for (int a = 0; a < K; ++a) cs[a * kShare + i] = cur.c[a][b0 + i];
    sid[i] = cur.id[b0 + i];
  }
  if (tid == 0) {
    begin[0][0] = 0;
    begin[0][1] = len;
    overflow = 0;
  }
  __syncthreads();
  uint32_t where[E];  // part << 16 | place of position e * T + tid, or kNone
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const uint32_t p = uint32_t(e) * T + tid;
    where[e] = p < len ? p : kNone;
  }
  Key k[E];
  int side = 0;
  bool dense = false;
  for (uint32_t j = 0; j <= levels; ++j) {
    const uint32_t d = (level + j) % K, parts = 1u << j, slot = kShare >> j;
    const uint32_t* bg = begin[side];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint32_t nd = where[e] >> 16, pl = where[e] & 0xffffu;
      if (where[e] == kNone) k[e] = Key::last();
      else if (j < levels) k[e] = Key::make(nd, OrdKey<A>::of(cs[d * kShare + pl]), pl);
      else k[e] = Key::make(nd, sid[pl], pl);
    }
    // positions e * T + tid to the networks' blocked order
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) ks.put(uint32_t(e) * T + tid, k[e]);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) k[e] = ks.get(tid * E + e);
    const int limit = dense ? int(kShare) : int(slot);
    warp_sort<Key, E>(k, tid & 31, limit);
    block_merges<Key, T, E, 64 * E>(k, ks, tid, limit);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) ks.put(tid * E + e, k[e]);
    __syncthreads();
    if (j == levels) break;
    if (tid < parts) {
      const uint32_t m = bg[tid + 1] - bg[tid], ideal = ideal_pivot(m);
      const uint32_t b = dense ? bg[tid] : tid * slot;  // where the part's keys begin
      uint32_t pivot = m;
      if (ideal < m) {
        const auto v = ks.get(b + ideal).key();
        const A value = OrdKey<A>::value(v);
        if (value == value) {  // a NaN at the ideal pivot splits nothing
          uint32_t x = 0, y = ideal;
          while (x < y) {  // first entry not below v
            const uint32_t h = (x + y) >> 1;
            if (ks.get(b + h).key() < v) x = h + 1;
            else y = h;
          }
          const uint32_t lt = x;
          x = ideal;
          y = m;
          while (lt == 0 && x < y) {  // first entry above v
            const uint32_t h = (x + y) >> 1;
            if (ks.get(b + h).key() > v) y = h;
            else x = h + 1;
          }
          pivot = lt > 0 ? lt : x;
          if (pivot < m) {
            const auto sk = ks.get(b + pivot).key();
            A stem = OrdKey<A>::value(sk);
            if (stem == A(0)) {  // the first zero in source order
              uint32_t best = 0xffffffffu;
              for (uint32_t i = pivot; i < m && ks.get(b + i).key() == sk; ++i) {
                const uint32_t pl = ks.get(b + i).place();
                if (sid[pl] <= best) {
                  best = sid[pl];
                  stem = cs[d * kShare + pl];
                }
              }
            }
            stems[(uint64_t(1) << (level + j)) + (uint64_t(node) << j) + tid] = stem;
          }
        }
      }
      begin[side ^ 1][2 * tid] = bg[tid];
      begin[side ^ 1][2 * tid + 1] = bg[tid] + pivot;
      if (tid == parts - 1) begin[side ^ 1][2 * parts] = len;
      if (pivot > slot / 2 || m - pivot > slot / 2) overflow = 1;
    }
    __syncthreads();
    // the next sub-level's positions
    const bool next_dense = overflow != 0;
    const uint32_t* nb = begin[side ^ 1];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint32_t p = uint32_t(e) * T + tid;
      uint32_t part, at, src;  // the part holding p, p's place in it, its key's position
      where[e] = kNone;
      if (next_dense) {
        if (p >= len) continue;
        uint32_t lo = 0, hi = 2 * parts;  // the last part that begins at or before p
        while (hi - lo > 1) {
          const uint32_t h = (lo + hi) >> 1;
          if (nb[h] <= p) lo = h;
          else hi = h;
        }
        part = lo;
        at = p - nb[part];
      } else {
        part = p / (slot / 2);
        at = p - part * (slot / 2);
        if (at >= nb[part + 1] - nb[part]) continue;
      }
      const uint32_t old = part >> 1, skip = (part & 1) ? nb[part] - nb[part - 1] : 0u;
      src = (dense ? bg[old] : old * slot) + skip + at;
      where[e] = (part << 16) | ks.get(src).place();
    }
    dense = next_dense;
    side ^= 1;
    __syncthreads();
  }
  const uint32_t leaves = 1u << levels, slot = kShare >> levels;
  const uint32_t* bg = begin[side];
  if (tid < leaves) {
    const uint64_t l = (uint64_t(node) << levels) + tid;
    leaf_b[l] = b0 + bg[tid];
    leaf_len[l] = bg[tid + 1] - bg[tid];
  }
  for (uint32_t p = tid; p < kShare; p += T) {
    uint32_t to = p;  // the place among the node's points
    if (dense) {
      if (p >= len) break;
    } else {
      const uint32_t part = p / slot, at = p - part * slot;
      if (at >= bg[part + 1] - bg[part]) continue;
      to = bg[part] + at;
    }
    const uint32_t pl = ks.get(p).place(), id = sid[pl];
    if constexpr (K == 3) {
      put_row<A>(arena, b0 + to, cs[pl], cs[kShare + pl], cs[2 * kShare + pl],
                 items ? items[id] : id);
    } else {
      ids[b0 + to] = id;
    }
  }
}

// The nodes above kShare points, in order, as fresh nodes: one block.
template <typename A>
__global__ void __launch_bounds__(1024) k_list_big(const Node<A>* __restrict__ nodes,
                                                   uint32_t count, Node<A>* __restrict__ out) {
  __shared__ uint32_t warp_n[32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t done = 0;
  for (uint32_t i0 = 0; i0 < count; i0 += 1024) {
    const uint32_t i = i0 + tid;
    const bool big = i < count && nodes[i].len > kShare;
    const unsigned m = __ballot_sync(FULL, big);
    if (lane == 0) warp_n[warp] = __popc(m);
    __syncthreads();
    uint32_t at = done + __popc(m & ((1u << lane) - 1u));
    for (uint32_t w = 0; w < 32; ++w) {
      at += w < warp ? warp_n[w] : 0u;
      done += warp_n[w];
    }
    if (big) out[at] = new_node<A>(nodes[i].index, nodes[i].b, nodes[i].len);
    __syncthreads();
  }
}

// ---- leaves -------------------------------------------------------------------------
// Encoded bytes of every leaf rounded up to 8 for the arena offsets, and the
// longest leaf.
template <typename A>
__global__ void k_leaf_sizes(int K, const uint32_t* __restrict__ nl, uint64_t leaves,
                             uint64_t* __restrict__ bytes, uint32_t* __restrict__ maxlen) {
  uint32_t longest = 0;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < leaves;
       i += uint64_t(gridDim.x) * blockDim.x) {
    uint64_t len = nl[i], total = 0;
    longest = max(longest, nl[i]);
    while (len) {
      const uint64_t w = len >= 32 ? 32 : len >= 8 ? 8 : len >= 4 ? 4 : len >= 2 ? 2 : 1;
      total += w * (K * sizeof(A) + sizeof(uint32_t));
      len -= w;
    }
    bytes[i] = (total + 7) & ~uint64_t(7);
  }
  longest = __reduce_max_sync(FULL, longest);
  if ((threadIdx.x & 31) == 0 && longest) atomicMax(maxlen, longest);
}

// Extents of every leaf as (offset / 8, len).  3-D rows sit at row_bytes() per
// point before them (in f32 those are the reference's offsets), other leaves at
// the reference's offsets; f64 rows keep the reference's beside them.
template <typename A, int K>
__global__ void k_leaf_extents(const uint32_t* __restrict__ nb, const uint32_t* __restrict__ nl,
                               const uint64_t* __restrict__ off, uint64_t leaves,
                               uint2* __restrict__ extents, uint2* __restrict__ src_extents) {
  for (uint64_t l = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; l < leaves;
       l += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t o = src_extents ? uint64_t(nb[l]) * row_bytes<A>() : off[l];
    extents[l] = make_uint2(uint32_t(o / 8), nl[l]);
    if (src_extents) src_extents[l] = make_uint2(uint32_t(off[l] / 8), nl[l]);
  }
}

// One warp per leaf: lane j writes point j's coordinates and item into its
// tile slot (or row).
template <typename A, int K>
__global__ void k_write_leaves(const A* __restrict__ pts, const uint32_t* __restrict__ items,
                               const uint32_t* __restrict__ sorted_ids,
                               const uint32_t* __restrict__ nb, const uint2* __restrict__ extents,
                               uint64_t leaves, uint8_t* __restrict__ arena) {
  const int lane = threadIdx.x & 31;
  for (uint64_t l = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; l < leaves;
       l += (uint64_t(gridDim.x) * blockDim.x) >> 5) {
    const uint64_t b = nb[l];
    const uint32_t len = extents[l].y;
    uint8_t* leaf = arena + uint64_t(extents[l].x) * 8;
    for (uint32_t p = lane; p < len; p += 32) {
      const uint32_t id = sorted_ids[b + p];
      uint32_t toff, w, i;
      tile_slot<A, K>(len, p, toff, w, i);
      A* col = reinterpret_cast<A*>(leaf + toff);
#pragma unroll
      for (int d = 0; d < K; ++d) col[d * w + i] = pts[uint64_t(id) * K + d];
      reinterpret_cast<uint32_t*>(leaf + toff + K * w * sizeof(A))[i] = items ? items[id] : id;
    }
  }
}

// Tiles <-> rows for the 3-D leaves held as rows on the device (RowLeaves),
// one warp per leaf: tiles at the reference's offsets (tex), rows at the
// device's (rex), the same point order.
template <typename A>
__device__ __forceinline__ void put_row(uint8_t* rows, uint32_t p, A x, A y, A z, uint32_t it) {
  if constexpr (sizeof(A) == 4) {
    reinterpret_cast<float4*>(rows)[p] = make_float4(x, y, z, __uint_as_float(it));
  } else {
    double2* r = reinterpret_cast<double2*>(rows) + 2 * size_t(p);
    r[0] = make_double2(x, y);
    r[1] = make_double2(z, __longlong_as_double((long long)it));  // item, then 4 zero bytes
  }
}

template <typename A>
__global__ void k_leaf_tiles_to_rows(const uint8_t* __restrict__ tiles, uint8_t* __restrict__ rows,
                                     const uint2* __restrict__ tex, const uint2* __restrict__ rex,
                                     uint64_t leaves) {
  const int lane = threadIdx.x & 31;
  for (uint64_t l = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; l < leaves;
       l += (uint64_t(gridDim.x) * blockDim.x) >> 5) {
    const uint2 te = tex[l];
    const size_t to = size_t(te.x) * 8, ro = size_t(rex[l].x) * 8;
    for (uint32_t p = lane; p < te.y; p += 32) {
      uint32_t toff, w, i;
      tile_slot_cols<A, 3>(te.y, p, toff, w, i);
      const A* col = reinterpret_cast<const A*>(tiles + to + toff);
      const uint32_t it = reinterpret_cast<const uint32_t*>(tiles + to + toff + 3 * w * sizeof(A))[i];
      put_row<A>(rows + ro, p, col[i], col[w + i], col[2 * w + i], it);
    }
  }
}

template <typename A>
__global__ void k_leaf_rows_to_tiles(const uint8_t* __restrict__ rows, uint8_t* __restrict__ tiles,
                                     const uint2* __restrict__ tex, const uint2* __restrict__ rex,
                                     uint64_t leaves) {
  const int lane = threadIdx.x & 31;
  for (uint64_t l = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; l < leaves;
       l += (uint64_t(gridDim.x) * blockDim.x) >> 5) {
    const uint2 te = tex[l];
    const size_t to = size_t(te.x) * 8, ro = size_t(rex[l].x) * 8;
    for (uint32_t p = lane; p < te.y; p += 32) {
      uint32_t toff, w, i;
      tile_slot_cols<A, 3>(te.y, p, toff, w, i);
      A c[3];
      uint32_t it;
      load_row<A, 3>(rows + ro, p, c, it);
      A* col = reinterpret_cast<A*>(tiles + to + toff);
      col[i] = c[0];
      col[w + i] = c[1];
      col[2 * w + i] = c[2];
      reinterpret_cast<uint32_t*>(tiles + to + toff + 3 * w * sizeof(A))[i] = it;
    }
  }
}

// Least item of every leaf, one warp per leaf (best_n_within leaves out leaves
// whose items are all too high).
template <typename A, int K>
__global__ void k_leaf_min(const uint8_t* __restrict__ arena, const uint2* __restrict__ extents,
                           uint64_t leaves, uint32_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  for (uint64_t l = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; l < leaves;
       l += (uint64_t(gridDim.x) * blockDim.x) >> 5) {
    const uint2 ex = extents[l];
    const uint8_t* leaf = arena + size_t(ex.x) * 8;
    uint32_t least = 0xffffffffu;
    for (uint32_t p = lane; p < ex.y; p += 32) {
      uint32_t off, w, i;
      tile_slot<A, K>(ex.y, p, off, w, i);
      least = min(least,
                  reinterpret_cast<const uint32_t*>(leaf + off + K * w * sizeof(A))[i]);
    }
    least = __reduce_min_sync(FULL, least);
    if (lane == 0) out[l] = least;
  }
}

// The subtrees of the `count` stems of one level, each the lesser of its two
// children's.
__global__ void k_node_min(uint32_t* __restrict__ m, uint32_t count) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint2 c = reinterpret_cast<const uint2*>(m)[count + i];
    m[count + i] = min(c.x, c.y);
  }
}
// The same for every level from `count` <= blockDim.x stems up to the root.
__global__ void __launch_bounds__(1024) k_top_min(uint32_t* m, uint32_t count) {
  for (; count; count /= 2) {
    if (threadIdx.x < count) {
      const uint32_t i = count + threadIdx.x;
      m[i] = min(m[2 * i], m[2 * i + 1]);
    }
    __syncthreads();
  }
}

inline unsigned blocks_for(uint64_t n, unsigned threads = 256) {
  const uint64_t b = (n + threads - 1) / threads;
  return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(b, 148ull * 64)));
}

int cuda_fail_b(cudaError_t e, const char* what) {
  return set_error(e == cudaErrorMemoryAllocation ? KGPU_ENOMEM : KGPU_ECUDA,
                   std::string(what) + ": " + cudaGetErrorString(e));
}

template <typename A, int K>
int build_on_device(const A* pts, const uint32_t* items, uint64_t n, cudaStream_t s,
                    DeviceTree& dt) {
  cudaError_t e;
  const uint64_t leaf_node_count = (n + kBucket - 1) / kBucket;
  uint32_t depth = 0;
  if (leaf_node_count >= 2)
    while ((uint64_t(1) << depth) < leaf_node_count) ++depth;
  const uint64_t leaves = n == 0 ? 0 : (uint64_t(1) << depth);
  const uint64_t stem_count = depth ? ((uint64_t(1) << (depth + 1)) + 7) / 8 * 8 : 0;
  dt.dtype = sizeof(A) == 8 ? KGPU_F64 : KGPU_F32;
  dt.dims = K;
  cudaGetDevice(&dt.device);
  dt.max_stem_level = depth ? int(depth) - 1 : -1;
  dt.leaf_count = uint32_t(leaves);
  dt.size = n;
  dt.stem_count = stem_count;
  dt.bh = 0;

  // the tree's arrays come from the stream-ordered pool, so rebuilding a tree of
  // similar size reuses cached memory
  dt.pooled = true;
  if ((e = scratch_alloc(&dt.stems, std::max<size_t>(16, stem_count * sizeof(A)), s)) !=
      cudaSuccess)
    return cuda_fail_b(e, "stems");
  A* stems = static_cast<A*>(dt.stems);
  auto no_stems = [&] {  // +inf = no split
    if (!stem_count) return;
    k_fill<A><<<blocks_for(stem_count), 256, 0, s>>>(stems, stem_count,
                                                     std::numeric_limits<A>::infinity());
    g_launches++;
  };
  no_stems();  // launched first: an idle GPU wakes up while the scratch is allocated

  // two sets of columns, which the level passes move the points between
  DevBuf col[2][K], idc[2];
  Columns<A, K> cols[2];
  for (int x = 0; x < 2; ++x) {
    for (int d = 0; d < K; ++d) {
      if ((e = col[x][d].alloc(n * sizeof(A), s)) != cudaSuccess)
        return cuda_fail_b(e, "construction scratch");
      cols[x].c[d] = col[x][d].template as<A>();
    }
    if ((e = idc[x].alloc(n * 4, s)) != cudaSuccess) return cuda_fail_b(e, "construction scratch");
    cols[x].id = idc[x].template as<uint32_t>();
  }
  // top levels: those above the nodes that k_finish takes
  const uint32_t last = std::min(depth, kShareLevels), top = depth - last;
  DevBuf nodes[2], hist, lb, ll, lids, lbytes, loff, scan_tmp, flags;
  // A level's table holds the top levels' nodes or, below them, the parts of
  // those that k_finish cannot take: fewer than n / kShare <= top_nodes, so
  // their parts fill two tables' worth at most.
  const uint64_t top_nodes = uint64_t(1) << top;
  auto hist_bytes = [](uint64_t count) {  // of the levels with up to `count` nodes
    uint64_t m = 4;
    for (uint64_t c = 1; c <= count; c <<= 1) m = std::max(m, (c << bins_log2_of(c)) * 4);
    return m;
  };
  if ((e = nodes[0].alloc(2 * top_nodes * sizeof(Node<A>), s)) != cudaSuccess ||
      (e = nodes[1].alloc(2 * top_nodes * sizeof(Node<A>), s)) != cudaSuccess ||
      (e = hist.alloc(hist_bytes(top_nodes), s)) != cudaSuccess ||
      (e = lb.alloc((leaves + 1) * 4, s)) != cudaSuccess ||
      (e = ll.alloc((leaves + 1) * 4, s)) != cudaSuccess ||
      (e = lids.alloc(K == 3 ? 16 : n * 4, s)) != cudaSuccess ||
      (e = lbytes.alloc((leaves + 1) * 8, s)) != cudaSuccess ||
      (e = loff.alloc((leaves + 1) * 8, s)) != cudaSuccess ||
      (e = scan_tmp.alloc(scan_tmp_bytes(leaves + 1), s)) != cudaSuccess ||
      (e = flags.alloc(16, s)) != cudaSuccess)
    return cuda_fail_b(e, "construction scratch");
  struct {
    uint32_t too_big, max_leaf, too_long;  // as in `flags`
  } seen = {0, 0, 0};
  int cur = 0, side = 0;  // which columns, which node table
  // The points in source order and one node.
  auto set_up = [&]() -> cudaError_t {
    cur = side = 0;
    k_columns<A, K><<<blocks_for(n), 256, 0, s>>>(pts, n, cols[0]);
    k_root<A><<<1, 1, 0, s>>>(nodes[0].template as<Node<A>>(), uint32_t(n));
    g_launches += 2;
    return cudaMemsetAsync(flags.p, 0, 16, s);
  };
  // The gaps above kLongGap that a level's partition left, once more through its
  // passes, with bins by key, until none is long (each round parts the bracket's
  // ends, so each makes a gap shorter).  The host waits for each round.  Only for
  // values spread over many exponents: 2^24 f32 points over 115 octaves 40 ms when one
  // block split every gap, 9.8 now, of which 4 for the first attempt.
  DevBuf gaps, want;
  auto split_gaps = [&](uint32_t count, int d, int bins_log2) -> cudaError_t {
    auto* nd = nodes[side].template as<Node<A>>();
    cudaError_t err = cudaSuccess;
    if (!gaps.p && ((err = gaps.alloc(2 * top_nodes * sizeof(Node<A>), s)) != cudaSuccess ||
                    (err = want.alloc(2 * top_nodes * 4, s)) != cudaSuccess))
      return err;
    auto* gp = gaps.template as<Node<A>>();
    uint32_t* at = want.template as<uint32_t>();
    const int x = cur ^ 1;  // the columns partitioned into
    const unsigned blocks = unsigned((n + 4095) / 4096), grid = std::min(count, 148u * 32);
    for (int round = 0; round < 12; ++round) {
      if ((err = cudaMemsetAsync(flags.as<uint32_t>() + 2, 0, 4, s)) != cudaSuccess) return err;
      k_list_gaps<A><<<blocks_for(count), 256, 0, s>>>(nd, count, gp, at,
                                                       flags.as<uint32_t>() + 2);
      ++g_launches;
      if ((err = cudaMemcpyAsync(&seen.too_long, flags.as<uint32_t>() + 2, 4,
                                 cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
          (err = cudaStreamSynchronize(s)) != cudaSuccess || !seen.too_long)
        return err;
      if ((err = cudaMemsetAsync(hist.p, 0, (uint64_t(count) << bins_log2) * 4, s)) != cudaSuccess)
        return err;
      k_bracket<A><<<grid, 256, 0, s>>>(cols[x].c[d], gp, count, 1u << bins_log2, at);
      k_histogram<A, true><<<blocks, 256, (size_t(1) << bins_log2) * 4, s>>>(
          cols[x].c[d], gp, count, uint32_t(n), 4096u, bins_log2, hist.template as<uint32_t>());
      k_find_bin<A><<<grid, 256, 0, s>>>(gp, count, hist.template as<uint32_t>(), 1u << bins_log2,
                                         at);
      k_partition<A, K, true><<<blocks, 256, 0, s>>>(cols[x], cols[cur], cols[x].c[d], gp, count,
                                                     uint32_t(n), 4096u, bins_log2);
      k_copy_gaps<A, K><<<blocks, 256, 0, s>>>(cols[cur], cols[x], gp, count, uint32_t(n), 4096u);
      k_take_gaps<A><<<blocks_for(count), 256, 0, s>>>(nd, count, gp);
      g_launches += 6;
    }
    return cudaGetLastError();
  };
  // One level: the node table nodes[side] (`count` nodes in order) and their
  // points in cols[cur] become the next level's.
  // `again`: with its long gaps split by all blocks.
  auto split_level = [&](uint32_t level, uint32_t count, bool again) -> cudaError_t {
    const int d = int(level % K);
    const int bins_log2 = bins_log2_of(count);
    auto* nd = nodes[side].template as<Node<A>>();
    cudaError_t err = cudaMemsetAsync(hist.p, 0, (uint64_t(count) << bins_log2) * 4, s);
    if (err != cudaSuccess) return err;
    // shares: whole waves of blocks on the first levels (few histogram
    // flushes), 8192 points and a few nodes at most on the others
    const uint64_t waves = (n + 148 * 8 - 1) / (148 * 8);
    const uint32_t share = uint32_t(count <= kTopNodes ? std::max<uint64_t>(8192, waves) : 8192);
    const unsigned blocks = unsigned((n + share - 1) / share);
    const int threads = count <= kTopNodes ? 1024 : 256;
    k_bracket<A><<<std::min(count, 148u * 32), 256, 0, s>>>(cols[cur].c[d], nd, count,
                                                            1u << bins_log2, nullptr);
    k_histogram<A><<<blocks, 256, (size_t(1) << bins_log2) * 4, s>>>(
        cols[cur].c[d], nd, count, uint32_t(n), share, bins_log2, hist.template as<uint32_t>());
    k_find_bin<A><<<std::min(count, 148u * 32), 256, 0, s>>>(
        nd, count, hist.template as<uint32_t>(), 1u << bins_log2, nullptr);
    const unsigned pblocks = unsigned((n + 4095) / 4096);
    k_partition<A, K><<<pblocks, 256, 0, s>>>(cols[cur], cols[cur ^ 1], cols[cur].c[d], nd, count,
                                              uint32_t(n), 4096u, bins_log2);
    if (again && (err = split_gaps(count, d, bins_log2)) != cudaSuccess) return err;
    k_select<A, K><<<std::min(count, 148u * 16), threads, 0, s>>>(
        cols[cur ^ 1], cols[cur], d, nd, count, stems + (uint64_t(1) << level),
        nodes[side ^ 1].template as<Node<A>>(), again ? nullptr : flags.as<uint32_t>() + 2);
    g_launches += 5;
    cur ^= 1;
    side ^= 1;
    return cudaGetLastError();
  };
  // the arena: 3-D leaves as rows, whose size is known; tiles once the leaves are
  const bool rows = RowLeaves<A, K>::value, moved = rows && sizeof(A) == 8;
  const uint64_t row_total = rows ? n * row_bytes<A>() : 0;
  auto make_rows = [&]() -> cudaError_t {
    const cudaError_t err = scratch_alloc(reinterpret_cast<void**>(&dt.arena), row_total + 16, s);
    return err != cudaSuccess ? err : cudaMemsetAsync(dt.arena + row_total, 0, 16, s);
  };
  uint64_t arena_bytes = 0;
  uint32_t last_len = 0;
  // leaf sizes, offsets and what the host needs of them
  auto leaf_tables = [&]() -> cudaError_t {
    cudaError_t err = cudaMemsetAsync(lbytes.as<uint64_t>() + leaves, 0, 8, s);
    if (err != cudaSuccess) return err;
    k_leaf_sizes<A><<<blocks_for(leaves), 256, 0, s>>>(K, ll.as<uint32_t>(), leaves,
                                                       lbytes.as<uint64_t>(),
                                                       flags.as<uint32_t>() + 1);
    g_launches++;
    if ((err = launch_exclusive_scan(lbytes.as<uint64_t>(), loff.as<uint64_t>(), leaves + 1,
                                     scan_tmp.p, s)) != cudaSuccess ||
        (err = cudaMemcpyAsync(&seen, flags.p, sizeof(seen), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (err = cudaMemcpyAsync(&arena_bytes, loff.as<uint64_t>() + leaves, 8,
                               cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (err = cudaMemcpyAsync(&last_len, ll.as<uint32_t>() + leaves - 1, 4,
                               cudaMemcpyDeviceToHost, s)) != cudaSuccess)
      return err;
    return cudaStreamSynchronize(s);
  };
  if (leaves) {
    auto kern = k_finish<A, K>;
    constexpr size_t smem = finish_smem<A, K>();
    // the levels from `level` on of the `count` nodes of nodes[side] that fit
    auto finish = [&](uint32_t level, uint32_t count) -> cudaError_t {
      const cudaError_t err =
          cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
      if (err != cudaSuccess) return err;
      kern<<<count, 256, smem, s>>>(cols[cur], nodes[side].template as<Node<A>>(), level,
                                    depth - level, stems, items, dt.arena, lids.as<uint32_t>(),
                                    lb.as<uint32_t>(), ll.as<uint32_t>(), flags.as<uint32_t>());
      g_launches++;
      return cudaGetLastError();
    };
    bool spread = false;  // a gap was too long: every level watches for such
    do {
      spread = seen.too_long != 0;
      if (spread) no_stems();
      // the leaves of nodes that k_finish leaves out have length 0 so far
      if ((e = set_up()) != cudaSuccess ||
          (e = cudaMemsetAsync(ll.p, 0, leaves * 4, s)) != cudaSuccess)
        return cuda_fail_b(e, "construction set-up");
      for (uint32_t level = 0; level < top; ++level)
        if ((e = split_level(level, 1u << level, spread)) != cudaSuccess)
          return cuda_fail_b(e, "construction levels");
      if (rows && !dt.arena && (e = make_rows()) != cudaSuccess)
        return cuda_fail_b(e, "tree arrays");
      if ((e = finish(top, uint32_t(top_nodes))) != cudaSuccess ||
          (e = leaf_tables()) != cudaSuccess)
        return cuda_fail_b(e, "the last levels");
    } while (seen.too_long && !spread);
    // Only the nodes that do not fit go on (a random 2^24-point f32 cloud has 24
    // of 8,192: 4.4 ms in all; 18.4 when every node went on and every leaf was
    // sorted again).
    bool more = false;
    for (uint32_t level = top, count = uint32_t(top_nodes); seen.too_big && level < depth;) {
      more = true;
      k_list_big<A><<<1, 1024, 0, s>>>(nodes[side].template as<Node<A>>(), count,
                                       nodes[side ^ 1].template as<Node<A>>());
      g_launches++;
      side ^= 1;
      count = seen.too_big;
      if ((e = split_level(level, count, true)) != cudaSuccess)
        return cuda_fail_b(e, "construction levels");
      ++level;
      count *= 2;
      if ((e = cudaMemsetAsync(flags.p, 0, 4, s)) != cudaSuccess ||
          (e = finish(level, count)) != cudaSuccess ||
          (e = cudaMemcpyAsync(&seen.too_big, flags.p, 4, cudaMemcpyDeviceToHost, s)) !=
              cudaSuccess ||
          (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return cuda_fail_b(e, "the last levels");
    }
    // a node that fits nowhere is a leaf above kShare points
    const bool overlong = seen.too_big != 0;
    if (more && !overlong && (e = leaf_tables()) != cudaSuccess)
      return cuda_fail_b(e, "leaf sizes");
    if (overlong || seen.max_leaf > 1024)
      return set_error(KGPU_EOVERFLOW,
                       "a leaf holds more than 1024 points (leaf scratch capacity, "
                       "leaf_view/mod.rs:18,58-65)");
    // the last leaf's bytes were counted rounded up to 8; the host arena ends at
    // the encoded end of the last leaf
    uint64_t raw = 0, rem = last_len;
    while (rem) {
      const uint64_t w = rem >= 32 ? 32 : rem >= 8 ? 8 : rem >= 4 ? 4 : rem >= 2 ? 2 : 1;
      raw += w * (K * sizeof(A) + sizeof(uint32_t));
      rem -= w;
    }
    arena_bytes = arena_bytes - ((raw + 7) & ~uint64_t(7)) + raw;
  }
  dt.leaf_bytes_len = arena_bytes;
  const uint64_t dev_bytes = moved ? row_total : arena_bytes;
  dt.max_leaf_len = seen.max_leaf;
  if ((!dt.arena &&
       (e = scratch_alloc(reinterpret_cast<void**>(&dt.arena), dev_bytes + 16, s)) !=
           cudaSuccess) ||
      (e = scratch_alloc(&dt.extents, std::max<size_t>(16, leaves * 8), s)) != cudaSuccess ||
      (e = scratch_alloc(reinterpret_cast<void**>(&dt.item_min),
                         std::max<size_t>(16, leaves * 8), s)) != cudaSuccess ||
      (moved && (e = scratch_alloc(&dt.src_extents, std::max<size_t>(16, leaves * 8), s)) !=
                    cudaSuccess))
    return cuda_fail_b(e, "tree arrays");
  if (!rows && (e = cudaMemsetAsync(dt.arena, 0, dev_bytes + 16, s)) != cudaSuccess)
    return cuda_fail_b(e, "arena");
  if (leaves) {
    k_leaf_extents<A, K><<<blocks_for(leaves), 256, 0, s>>>(
        lb.as<uint32_t>(), ll.as<uint32_t>(), loff.as<uint64_t>(), leaves,
        static_cast<uint2*>(dt.extents), static_cast<uint2*>(dt.src_extents));
    g_launches++;
    if (!rows) {
      k_write_leaves<A, K><<<blocks_for(leaves * 32), 256, 0, s>>>(
          pts, items, lids.as<uint32_t>(), lb.as<uint32_t>(), static_cast<uint2*>(dt.extents),
          leaves, dt.arena);
      g_launches++;
    }
  }
  if ((e = cudaGetLastError()) != cudaSuccess || (e = fill_item_min(dt, s)) != cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return cuda_fail_b(e, "writing the leaves");
  dt.device_bytes = std::max<size_t>(16, stem_count * sizeof(A)) + dev_bytes + 16 +
                    leaves * 8 * (moved ? 3 : 2);
  return KGPU_OK;
}

}  // namespace

cudaError_t fill_item_min(const DeviceTree& dt, cudaStream_t s) {
  if (dt.leaf_count == 0) return cudaSuccess;
  const unsigned grid = blocks_for(uint64_t(dt.leaf_count) * 32);
  auto run = [&](auto kern) {
    kern<<<grid, 256, 0, s>>>(dt.arena, static_cast<const uint2*>(dt.extents), dt.leaf_count,
                              dt.item_min + dt.leaf_count);
    g_launches++;
    if (dt.scalar_walk()) return cudaGetLastError();
    // subtrees, from the leaves up: a launch per level, the last ones in one block
    uint32_t count = dt.leaf_count / 2;  // a power of two
    for (; count > 1024; count /= 2) {
      k_node_min<<<blocks_for(count), 256, 0, s>>>(dt.item_min, count);
      g_launches++;
    }
    if (count) {
      k_top_min<<<1, 1024, 0, s>>>(dt.item_min, count);
      g_launches++;
    }
    return cudaGetLastError();
  };
  const bool f64 = dt.dtype == KGPU_F64;
  switch (dt.dims) {
    case 1: return f64 ? run(k_leaf_min<double, 1>) : run(k_leaf_min<float, 1>);
    case 2: return f64 ? run(k_leaf_min<double, 2>) : run(k_leaf_min<float, 2>);
    case 3: return f64 ? run(k_leaf_min<double, 3>) : run(k_leaf_min<float, 3>);
    case 4: return f64 ? run(k_leaf_min<double, 4>) : run(k_leaf_min<float, 4>);
  }
  return cudaErrorInvalidValue;
}

cudaError_t convert_leaf_layout(const DeviceTree& dt, const uint8_t* src, uint8_t* dst,
                                bool to_rows, cudaStream_t s) {
  if (dt.leaf_count == 0) return cudaSuccess;
  const unsigned grid = blocks_for(uint64_t(dt.leaf_count) * 32);
  const uint2* rex = static_cast<const uint2*>(dt.extents);
  const uint2* tex = dt.src_extents ? static_cast<const uint2*>(dt.src_extents) : rex;
  if (dt.dtype == KGPU_F64) {
    if (to_rows) k_leaf_tiles_to_rows<double><<<grid, 256, 0, s>>>(src, dst, tex, rex, dt.leaf_count);
    else k_leaf_rows_to_tiles<double><<<grid, 256, 0, s>>>(src, dst, tex, rex, dt.leaf_count);
  } else {
    if (to_rows) k_leaf_tiles_to_rows<float><<<grid, 256, 0, s>>>(src, dst, tex, rex, dt.leaf_count);
    else k_leaf_rows_to_tiles<float><<<grid, 256, 0, s>>>(src, dst, tex, rex, dt.leaf_count);
  }
  g_launches++;
  return cudaGetLastError();
}

namespace {

template <typename A>
int build_any_dims(int K, const void* pts, const uint32_t* items, uint64_t n, cudaStream_t s,
                   DeviceTree& dt) {
  const A* p = static_cast<const A*>(pts);
  switch (K) {
    case 1: return build_on_device<A, 1>(p, items, n, s, dt);
    case 2: return build_on_device<A, 2>(p, items, n, s, dt);
    case 3: return build_on_device<A, 3>(p, items, n, s, dt);
    case 4: return build_on_device<A, 4>(p, items, n, s, dt);
  }
  return set_error(KGPU_EUNSUPPORTED, "dims must be 1..4");
}

}  // namespace
}  // namespace kgpu

using namespace kgpu;

extern "C" {

int32_t kgpu_tree_build(int32_t dtype, uint32_t dims, const void* points, const uint32_t* items,
                        uint64_t n, void* stream, kgpu_tree** out) {
  if (!out) return set_error(KGPU_EINVAL, "out is NULL");
  *out = nullptr;
  if (dims < 1 || dims > uint32_t(kMaxDims)) return set_error(KGPU_EUNSUPPORTED, "dims must be 1..4");
  if (dtype != KGPU_F32 && dtype != KGPU_F64)
    return set_error(KGPU_EINVAL, "dtype must be KGPU_F32 or KGPU_F64");
  if (n > 0 && !points) return set_error(KGPU_EINVAL, "points is NULL");
  if (n >= (uint64_t(1) << 31)) return set_error(KGPU_EOVERFLOW, "2^31 points or more");
  auto* t = new (std::nothrow) kgpu_tree();
  if (!t) return set_error(KGPU_ENOMEM, "host allocation failed");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int st = dtype == KGPU_F64
                     ? build_any_dims<double>(int(dims), points, items, n, s, t->dt)
                     : build_any_dims<float>(int(dims), points, items, n, s, t->dt);
  if (st != KGPU_OK) {
    cudaStreamSynchronize(s);
    release_tree_arrays(t->dt);
    delete t;
    return st;
  }
  *out = t;
  return KGPU_OK;
}

int32_t kgpu_tree_read_layout(const kgpu_tree* t, void* stems, uint8_t* leaf_bytes,
                              uint64_t* extents, void* stream) {
  if (!t) return set_error(KGPU_EINVAL, "NULL tree");
  const DeviceTree& dt = t->dt;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t sa = dt.dtype == KGPU_F64 ? 8 : 4;
  std::vector<uint32_t> ex(2 * size_t(dt.leaf_count));
  cudaError_t e;
  // leaves held as rows go back to the reference's tiles first
  DevBuf tiles;
  const uint8_t* arena = dt.arena;
  if (leaf_bytes && dt.leaf_bytes_len && dt.dims == 3) {
    if ((e = tiles.alloc(dt.leaf_bytes_len, s)) != cudaSuccess ||
        (e = cudaMemsetAsync(tiles.p, 0, dt.leaf_bytes_len, s)) != cudaSuccess ||
        (e = convert_leaf_layout(dt, dt.arena, tiles.as<uint8_t>(), false, s)) != cudaSuccess)
      return cuda_fail_b(e, "reading the layout");
    arena = tiles.as<uint8_t>();
  }
  if ((stems && dt.stem_count &&
       (e = cudaMemcpyAsync(stems, dt.stems, dt.stem_count * sa, cudaMemcpyDeviceToHost, s)) !=
           cudaSuccess) ||
      (leaf_bytes && dt.leaf_bytes_len &&
       (e = cudaMemcpyAsync(leaf_bytes, arena, dt.leaf_bytes_len, cudaMemcpyDeviceToHost, s)) !=
           cudaSuccess) ||
      (dt.leaf_count &&
       (e = cudaMemcpyAsync(ex.data(), dt.src_extents ? dt.src_extents : dt.extents,
                            ex.size() * 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess))
    return cuda_fail_b(e, "reading the layout");
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail_b(e, "reading the layout");
  if (extents)
    for (size_t l = 0; l < dt.leaf_count; ++l) {
      extents[2 * l] = uint64_t(ex[2 * l]) * 8;
      extents[2 * l + 1] = ex[2 * l + 1];
    }
  return KGPU_OK;
}

}  // extern "C"
