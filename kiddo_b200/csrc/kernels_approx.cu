// kernels_approx.cu — approx nearest_one on 2-D and 3-D trees, queries in the
// caller's order (batches grouped by leaf run k_tfixed).
#include "kgpu_launch_impl.cuh"

namespace kgpu {
namespace {

// The first lane that holds the warp's least d, which is +0 or more; 0 where all
// are +inf or NaN.
__device__ __forceinline__ unsigned warp_first_min(float d) {
  const unsigned bits = __float_as_uint(d);
  const unsigned m = __reduce_min_sync(FULL, bits);
  return unsigned(__ffs(__ballot_sync(FULL, bits == m)) - 1);
}
__device__ __forceinline__ unsigned warp_first_min(double d) {
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(d));
  const unsigned hi = unsigned(bits >> 32), lo = unsigned(bits);
  const unsigned mh = __reduce_min_sync(FULL, hi);
  const unsigned ml = __reduce_min_sync(FULL, hi == mh ? lo : 0xffffffffu);
  return unsigned(__ffs(__ballot_sync(FULL, hi == mh && lo == ml)) - 1);
}

// approx nearest_one (one straight descent, one leaf): each lane descends for its
// own query, then the warp scans the 32 leaves one after another, lane p on point
// p, kOwners of them in flight.  The least distance is a reduction of its bits
// (distances are +0 or more; NaN bits lie above those of +inf, which nothing
// reports), and the first lane that holds it names the item: the first minimum
// in leaf order, as the sequential `d < best` keeps.
//
// What bounds it: the latency of the leaves, half of them from HBM.  Queries are taken
// in the caller's order, so results and queries stream, and a leaf of about 30 f32
// rows is one 480-byte read: 7.7 GB for 16M random queries of a 16M-point clustered
// tree, 1.71 ms, of which the L2 serves half (8M of 8M: 2.0 GB of DRAM reads, 51% of
// issue slots, 6.9 warps waiting on loads per issue).  Grouping the
// batch by leaf, with a leaf read once for a warp's 32 queries, took 2.72 ms:
// 0.72 of sorting, and scattered reads of queries and writes of results.
template <typename A, int K, typename M>
__global__ void __launch_bounds__(256) k_approx(TreeView<A> tv0, Batch<A> b,
                                                A* __restrict__ out_d,
                                                uint32_t* __restrict__ out_i,
                                                uint32_t* __restrict__ out_c,
                                                unsigned long long* __restrict__ stats) {
  constexpr int kOwners = sizeof(A) == 4 ? 8 : 4;
  const int lane = threadIdx.x & 31;
  const uint64_t nq = b.count();
  const uint64_t step = uint64_t(gridDim.x) * blockDim.x;
  TravStats st;
  for (uint64_t w0 = uint64_t(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u); w0 < nq;
       w0 += step) {
    const bool mine = w0 + lane < nq;
    uint64_t qi = 0;
    A q[K];
#pragma unroll
    for (int d = 0; d < K; ++d) q[d] = A(0);
    const uint8_t* base = tv0.arena;
    uint32_t len = 0;
    if (mine) {
      qi = b.order ? uint64_t(b.order[w0 + lane]) : w0 + lane;
      const TreeView<A> tv = b.tree(tv0, qi);
      b.query(qi, q);
      if (tv.leaf_count > 0) {
        const uint2 ex = __ldg(tv.extents + straight_leaf<A, K>(tv, q));
        base = tv.arena + size_t(ex.x) * 8;
        len = ex.y;
        st.points += len;
        st.stems += uint32_t(tv.max_stem_level + 1);
        st.leaves += 1;
      }
    }
    A best = inf_of<A>();
    uint32_t item = 0;
    for (int o0 = 0; o0 < 32; o0 += kOwners) {
      A c[kOwners][K];
      uint32_t it[kOwners], n[kOwners];
#pragma unroll
      for (int j = 0; j < kOwners; ++j) {
        n[j] = shfl(len, o0 + j);
        const uint8_t* leaf = reinterpret_cast<const uint8_t*>(
            __shfl_sync(FULL, reinterpret_cast<unsigned long long>(base), o0 + j));
        it[j] = 0;
        if (uint32_t(lane) < n[j]) load_point<A, K>(leaf, n[j], lane, c[j], it[j]);
      }
#pragma unroll
      for (int j = 0; j < kOwners; ++j) {
        A oq[K];
#pragma unroll
        for (int d = 0; d < K; ++d) oq[d] = shfl(q[d], o0 + j);
        A d = inf_of<A>();
        if (uint32_t(lane) < n[j]) d = point_dist<M, A, K>(c[j], oq);
        const unsigned first = warp_first_min(d);
        const uint32_t ci = shfl(it[j], int(first & 31u));
        const A cd = shfl(d, int(first & 31u));
        if (lane == o0 + j && cd < best) {
          best = cd;
          item = ci;
        }
      }
    }
    // leaves longer than a warp (many equal points)
    for (unsigned lm = __ballot_sync(FULL, len > 32); lm; lm &= lm - 1) {
      const int o = __ffs(lm) - 1;
      const uint32_t n = shfl(len, o);
      const uint8_t* leaf = reinterpret_cast<const uint8_t*>(
          __shfl_sync(FULL, reinterpret_cast<unsigned long long>(base), o));
      A oq[K];
#pragma unroll
      for (int d = 0; d < K; ++d) oq[d] = shfl(q[d], o);
      for (uint32_t c0 = 32; c0 < n; c0 += 32) {
        A c[K], d = inf_of<A>();
        uint32_t it = 0;
        if (c0 + lane < n) {
          load_point<A, K>(leaf, n, c0 + lane, c, it);
          d = point_dist<M, A, K>(c, oq);
        }
        const unsigned first = warp_first_min(d);
        const uint32_t ci = shfl(it, int(first & 31u));
        const A cd = shfl(d, int(first & 31u));
        if (lane == o && cd < best) {
          best = cd;
          item = ci;
        }
      }
    }
    if (mine) {
      out_d[qi] = best;
      out_i[qi] = item;
      if (out_c) out_c[qi] = 1;
    }
  }
  if (stats) flush_stats(stats, st);
}

}  // namespace

template <typename A>
cudaError_t launch_approx(const DeviceTree& t, const QueryLaunch& q) {
  const TreeView<A> tv = make_view<A>(t);
  const Batch<A> b = make_batch<A>(q);
  return with_dims(t.dims, [&](auto kk) -> cudaError_t {
    constexpr int K = decltype(kk)::value;
    if constexpr (!thread_engine_dims(K)) {
      return cudaErrorInvalidValue;
    } else {
      return with_metric(q.metric, [&](auto m) {
        auto kern = k_approx<A, K, decltype(m)>;
        kern<<<grid_for(kern, 0, (q.nq + 31) / 32), 256, 0, q.stream>>>(
            tv, b, static_cast<A*>(q.out_d), q.out_i, q.out_c, q.stats);
        g_launches++;
        return cudaGetLastError();
      });
    }
  });
}
template cudaError_t launch_approx<float>(const DeviceTree&, const QueryLaunch&);
template cudaError_t launch_approx<double>(const DeviceTree&, const QueryLaunch&);

}  // namespace kgpu
