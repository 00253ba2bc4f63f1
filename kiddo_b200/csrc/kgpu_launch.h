// kgpu_launch.h — host-side launch interface between the API and the kernels.
#pragma once

#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/kiddo_gpu.h"

namespace kgpu {

struct DeviceTree {
  int dtype = 0;
  int dims = 0;
  int device = 0;
  void* stems = nullptr;       // A[stem_count]
  uint8_t* arena = nullptr;    // leaf bytes
  void* extents = nullptr;     // uint2 (offset/8, len) [leaf_count]
  int max_stem_level = -1;
  uint32_t leaf_count = 0;
  uint64_t size = 0;
  uint64_t stem_count = 0;
  uint64_t leaf_bytes_len = 0;
  uint64_t max_leaf_len = 0;
  size_t device_bytes = 0;
  uint32_t bh = 0;             // 0: Eytzinger stems; 3 or 4: Donnelly<bh>
  // Mapped stem/leaf resolution: u32 leaf of each stem index from map_min
  // (0xffffffff: not terminal) on the device, or null (arithmetic)
  uint32_t* leaf_map = nullptr;
  // least item of each leaf (0xffffffff: empty) at [leaf_count, 2 leaf_count);
  // below, for arithmetic Eytzinger trees, of each stem's subtree at its index
  uint32_t* item_min = nullptr;
  uint64_t map_min = 0;
  uint32_t map_len = 0;
  // the kernels' scalar backtracking walk (Donnelly stems or Mapped resolution)
  // rather than the Eytzinger arithmetic DFS
  bool scalar_walk() const { return bh != 0 || leaf_map != nullptr; }
  bool pooled = false;         // arrays from the stream-ordered pool (device-built trees)
  // f64 3-D leaves are 32-byte rows with offsets of their own: the reference
  // layout's extents, uint2 (offset / 8, len), for read-back; null otherwise
  void* src_extents = nullptr;
  // stored points of query results (kgpu_tree_project), built on first use:
  // the entries' points in iteration order, and (item, rank) sorted by item
  void* iter_points = nullptr;
  uint32_t* sorted_items = nullptr;
  uint32_t* sorted_ranks = nullptr;
  int items_distinct = -1;     // -1: not checked yet; 0: two entries share an item; 1: distinct
  // per-axis bounds of the stored points, measured on first use by periodic
  // queries (kgpu_periodic_fast.cu): -1 not measured, 0 unusable (no points,
  // or a NaN coordinate), 1 measured
  mutable int point_bounds = -1;
  mutable double point_lo[4] = {0, 0, 0, 0}, point_hi[4] = {0, 0, 0, 0};
};

struct QueryLaunch {
  int family = 0;     // kgpu_family
  int metric = 0;     // kgpu_metric
  int k = 1;
  double radius = 0;
  bool exclusive = false;
  bool sorted = true;
  const void* queries = nullptr;  // device, nq * dims values of A
  const uint32_t* order = nullptr;  // optional processing order (device)
  uint64_t nq = 0;
  void* out_d = nullptr;
  uint32_t* out_i = nullptr;
  uint32_t* out_c = nullptr;
  unsigned long long* stats = nullptr;  // optional [stems, leaves, points] totals
  uint32_t chunk = 0;             // queries handed to a warp at a time (lane-refilled drivers)
  int refill = 0;                 // idle lanes a warp waits for before refilling them; 0: defaults
  int engine = 0;                 // 0 auto, 1 warp per query, 2 thread per query,
                                  // 3 thread walks with warp-cooperative leaf scans
  bool periodic = false;          // periodic boundary conditions
  double box[4] = {0, 0, 0, 0};   // periodic box (converted to A)
  // batches over many trees (see kgpu_forest_*): device arrays, or null
  const void* forest = nullptr;          // TreeView<A>[n_trees]
  const uint32_t* tree_of = nullptr;     // tree of each query
  uint32_t n_trees = 0;
  const uint64_t* leaf_base = nullptr;   // first global leaf number of each tree
  uint64_t total_leaves = 0;             // leaves of all trees (spatial order)
  const void* radii = nullptr;           // per-query radius (A), or null
  unsigned long long* work = nullptr;    // work-queue counter (zeroed), or null
  const unsigned long long* nq_dev = nullptr;  // device count bounding nq
  int32_t dev_line = 0;  // device counts this launch is for (Batch::dev_line)
  uint64_t capacity = ~uint64_t(0);      // fill pass: hits that fit the output
  int* status = nullptr;                 // fill pass: set to KGPU_EOVERFLOW on mismatch
  cudaStream_t stream = nullptr;
};

// process-wide count of kernel launches made by this library
extern std::atomic<uint64_t> g_launches;

// QueryLaunch::engine from a query's KGPU_FLAG_ENGINE_* bits.
inline int engine_of(uint32_t flags) {
  return (flags & KGPU_FLAG_ENGINE_WARP) ? 1 : (flags & KGPU_FLAG_ENGINE_THREAD) ? 2
         : (flags & KGPU_FLAG_ENGINE_COOP) ? 3 : 0;
}

// The launch knobs of kgpu_query_desc::tuning (KGPU_TUNE_*); 0 fields keep
// the defaults (make_batch).
inline void apply_tuning(uint32_t tuning, QueryLaunch& q) {
  const uint32_t refill = tuning & 0x3fu;
  const uint32_t chunk_log2 = (tuning >> 8) & 0xfu;
  if (refill >= 1 && refill <= 32) q.refill = int(refill);
  if (chunk_log2 >= 5 && chunk_log2 <= 10) q.chunk = 1u << chunk_log2;
}

// The engine of a batch that asks for none: small batches of 2-D and 3-D trees
// take the warp engine.  A thread walks its query alone, so a batch too small
// to fill the GPU with threads takes as long as one thread's walk (50 us to 1
// ms); a warp answers a query in about a twentieth of that, and the engines
// meet where the warps' throughput reaches the thread's latency: earlier over
// uniform points, later over clustered ones, whose slowest walks are longer.
// The lines lie between.  Measured, 1M-point trees, uniform; clustered (thread
// or cooperative / warp engine, us):
//   nearest_one f32 24576 queries 73/68; 127/66, 49152 79/125; 129/105
//   nearest_n f32 k = 8 32768 131/153; 360/185, 49152 137/220; 372/239
//     k = 16 32768 198/198; 473/233, 65535 217/366; 500/394
//     k = 32 40000 376/332; 434/386, 65535 384/537; 455/565
//   nearest_n f64 k = 16 40000 335/294; 382/274, 65535 345/458; 406/432
//     k = 32 49152 540/495; 583/481, 65535 546/639; 587/605
//   best_n f32 40000 155/147; 126/106, 49152 156/175; 132/128
//   within f32 3-D (one walk) 16384 239/242; 200/190, 24576 242/286; 202/225,
//     2-D (two walks) 40000 287/276
//   periodic nearest_n f32 k = 16 32768 369/370; 468/388, f64 k = 32 24576
//     766/593; 913/632, 32768 772/798; 911/803; within f32 24576 439/441;
//     354/308, f64 16384 567/530; 412/379
//   f32 k = 64 49152 1164/1334; 1871/1402
// f64 lists above 32 entries leave two blocks of threads per SM, fewer the longer
// they are: the lines run from 65536 queries at k = 33 over 524288 at 40 to none
// from 45 on (thread / warp engine, ms, uniform; sphere; clustered: k = 33 100k
// queries 1.65/1.88; 1.46/1.61; 2.12/2.10, 2M 21.4/34.4; 17.1/30.0; 24.5/37.5, k =
// 40 500k 10.8/10.8; 8.9/9.5; 12.6/12.0, 2M 38.8/41.9; 29.9/37.4; 43.4/46.4, k = 48
// 2M 52.4/48.0; 39.4/43.2; 57.5/53.6, k = 64 2M 80.7/60.5; 58.4/54.1; 87.2/67.3).
// Explicit engines, Donnelly and Mapped trees (thread walks
// only) and lists kept in output rows are not touched.
inline int engine_for(const DeviceTree& t, const QueryLaunch& q) {
  if (q.engine != 0 || t.scalar_walk() || (t.dims != 2 && t.dims != 3)) return q.engine;
  const uint64_t k = uint64_t(q.k > 0 ? q.k : 1);
  const bool f64 = t.dtype == KGPU_F64;
  uint64_t below = 0;
  switch (q.family) {
    case KGPU_NEAREST_ONE:
      below = 28672;
      break;
    case KGPU_NEAREST_N:
    case KGPU_NEAREST_N_WITHIN:
      if (q.periodic) below = k <= 32 ? (f64 ? 22528 : 28672) + 384 * k : 0;
      else if (k > 32 && f64) below = k < 45 ? uint64_t(65536) << (k - 33) * 3 / 7 : ~uint64_t(0);
      else if (k > 32) below = 32768 + 512 * (k - 32);
      else if (k > (f64 ? 13 : 20)) below = f64 ? 57344 : 49152;
      else below = 32768 + 768 * k;
      break;
    case KGPU_BEST_N_WITHIN:
      below = 40960;
      break;
    case KGPU_WITHIN:
    case KGPU_WITHIN_UNSORTED:
      below = q.periodic ? (f64 ? 18432 : 24576) : t.dims == 3 ? 16384 : 40960;
      break;
    default:  // approx: one leaf per query, the thread engine's at every size
      break;
  }
  return q.nq < below ? 1 : q.engine;
}

// Whether a large batch that does not ask for leaf-grouped order gets it.  Not
// f32 approx: a leaf is one 480-byte read there, and reading it again for each
// query costs less than the sort and the scattered queries and results (16M
// queries of a 16M-point tree 1.71 ms against 2.72, 8M of 100k points 0.55
// against 0.99, 2-D 8M of 8M 0.95 against 1.11).  f64 leaves are twice that and
// do not (8M of 8M 1.58 against 1.28 ms, 2-D 4M of 4M 0.60 against 0.55).
inline bool order_pays(const DeviceTree& t, const QueryLaunch& q, uint32_t flags) {
  return (flags & KGPU_FLAG_SPATIAL_ORDER) || q.family != KGPU_APPROX_NEAREST_ONE ||
         t.dtype == KGPU_F64 || q.engine == 1 || (t.dims != 2 && t.dims != 3);
}

// Fixed-size families: dispatches to the thread engine (2-D/3-D trees) or the
// warp engine (everything else, periodic included).
template <typename A> cudaError_t launch_fixed(const DeviceTree& t, const QueryLaunch& q);

// Periodic sorted nearest_n over one tree through a plain walk where the box's
// faces cannot change a row, and the periodic walk for the other rows
// (kgpu_periodic_fast.cu).  `handled` is false, with nothing launched, where
// it does not apply; the caller then launches the periodic walk itself.
template <typename A>
cudaError_t periodic_fast(const DeviceTree& t, const QueryLaunch& q, bool& handled);
template <typename A> cudaError_t launch_wfixed(const DeviceTree& t, const QueryLaunch& q);
template <typename A> cudaError_t launch_tfixed(const DeviceTree& t, const QueryLaunch& q);
// approx nearest_one on 2-D and 3-D trees of either stem order, queries in the
// caller's order (kernels_approx.cu).
template <typename A> cudaError_t launch_approx(const DeviceTree& t, const QueryLaunch& q);
// Lists of any length held in the output rows (kernels_*_rows.cu).
template <typename A> cudaError_t launch_trow(const DeviceTree& t, const QueryLaunch& q);
// Donnelly-stem kernels, defined in their own translation units
// (kernels_f32_donnelly.cu, kernels_f64_donnelly.cu); the last argument only
// selects the coordinate type.
cudaError_t launch_tfixed_donnelly(const DeviceTree& t, const QueryLaunch& q, float);
cudaError_t launch_tfixed_donnelly(const DeviceTree& t, const QueryLaunch& q, double);
cudaError_t launch_within_donnelly(const DeviceTree& t, const QueryLaunch& q, uint64_t* counts,
                                   const uint64_t* offsets, float);
cudaError_t launch_within_donnelly(const DeviceTree& t, const QueryLaunch& q, uint64_t* counts,
                                   const uint64_t* offsets, double);
template <typename A> cudaError_t launch_within_count(const DeviceTree& t, const QueryLaunch& q,
                                                       uint64_t* counts);
template <typename A> cudaError_t launch_within_fill(const DeviceTree& t, const QueryLaunch& q,
                                                      const uint64_t* offsets);
// Records of the hits that a counting pass saw (kgpu_hits.cuh): per leaf chunk
// with hits its rows' address, the mask of hits and the hits of its query before
// it, and the query.  `count` may pass `cap`; records beyond are lost.
struct HitRecords {
  uint4* leaf = nullptr;
  uint32_t* query = nullptr;
  unsigned long long* count = nullptr;
  uint64_t cap = 0;
};
// 3-D arithmetic trees (rows, ThreadWalk), no periodic box.
template <typename A> cudaError_t launch_within_record(const DeviceTree& t, const QueryLaunch& q,
                                                       uint64_t* counts, const HitRecords& rec);
template <typename A> cudaError_t launch_place_hits(const QueryLaunch& q, const uint64_t* offsets,
                                                    const HitRecords& rec, uint64_t n);
// Processing order grouped by straight-descent leaf.  `scratch` must hold
// spatial_order_scratch_bytes(t, nq) bytes; order[nq] receives query indices.
size_t spatial_order_scratch_bytes(const DeviceTree& t, const QueryLaunch& q);
template <typename A> cudaError_t launch_spatial_order(const DeviceTree& t, const QueryLaunch& q,
                                                       uint32_t* order, void* scratch);

// Stable sort of every CSR segment by distance; scratch holds total entries.
// Segments are clamped to the first `capacity` entries.
template <typename A> cudaError_t launch_seg_sort(const uint64_t* offsets, uint64_t nq,
                                                  uint64_t capacity, A* d, uint32_t* it,
                                                  A* scratch_d, uint32_t* scratch_i,
                                                  cudaStream_t s);

// offsets[0..n] = exclusive prefix sum of counts[0..n) (offsets[n] = total).
// `counts` and `offsets` may alias.  tmp needs scan_tmp_bytes(n) bytes.
size_t scan_tmp_bytes(uint64_t n);
cudaError_t launch_exclusive_scan(const uint64_t* counts, uint64_t* offsets, uint64_t n,
                                  void* tmp, cudaStream_t s);

int sm_count();

// Fills dt.item_min from the stored leaves.
cudaError_t fill_item_min(const DeviceTree& dt, cudaStream_t s);

// Re-encodes a tree's 3-D leaves between the reference's tiles (at the
// offsets of dt.src_extents, or of dt.extents when that is null) and the
// device's rows (at the offsets of dt.extents).
cudaError_t convert_leaf_layout(const DeviceTree& dt, const uint8_t* src, uint8_t* dst,
                                bool to_rows, cudaStream_t s);

}  // namespace kgpu
