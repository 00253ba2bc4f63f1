// kgpu_hits.cuh — radius queries in one walk: the counting pass keeps where its
// hits are, and the filling pass places them from that.
//
// The two-pass form walks every tree twice, though the second walk only finds
// again what the first one saw.  Here the counting pass (k_twithin_record)
// appends a record per leaf chunk that holds hits: the chunk's address, the
// mask of its points within the radius, the query and the hits it had before.
// k_place_hits then takes 32 records per warp, recomputes the distances of the
// masked points (the same operations, the same bits) and writes them at the
// query's offset, never past the end of the query's row or of the outputs.  Records cost 20 bytes per 32 points with a hit; a batch with
// more than its buffer holds is filled by the second walk instead.
//
// What bounds it: instruction issue in the counting walk; in the placing pass the
// scattered short writes (a record's hits are about 6 words in each output).
#pragma once

#include "kgpu_kernels.cuh"

namespace kgpu {

// CWithin's counting leaf scan, appending records.  A warp takes room for
// kBatch records at a time, so most appends touch no shared counter.
template <typename A, int K, typename M, bool kExclusive>
struct CWithinRecord {
  static constexpr bool kPruneOnEqual = kExclusive;
  static constexpr uint32_t kBatch = 64;
  A radius;
  uint32_t count;  // a tree holds fewer than 2^32 points
  HitRecords rec;
  unsigned long long at;  // the warp's next record
  uint32_t left;          // of the room it took
  __device__ explicit CWithinRecord(const HitRecords& r)
      : radius(A(0)), count(0), rec(r), at(0), left(0) {}
  __device__ __forceinline__ A max_dist() const { return radius; }
  __device__ __forceinline__ bool unbounded_start() const { return radius == inf_of<A>(); }

  __device__ __forceinline__ void leaf(int o, uint64_t qi, const CoopLeaf<A, K>& L, int lane) {
    uint32_t had = 0;  // the owner's hits so far, and its query: read for the first record
    uint32_t query = 0;
    bool hit = false;
    const A orad = shfl(radius, o);
    for (uint32_t c0 = 0; c0 < L.len; c0 += 32) {
      const uint32_t p = c0 + lane;
      bool pass = false;
      if (p < L.len) {
        uint32_t it;
        const A d = coop_point<A, K>(L, p, it, CartesianDist<A, K, M>());
        pass = kExclusive ? (d < orad) : (d <= orad);
      }
      const unsigned m = __ballot_sync(FULL, pass);
      if (!m) continue;
      if (!hit) {
        had = shfl(count, o);
        query = shfl(uint32_t(qi), o);
        hit = true;
      }
      if (left == 0) {
        if (lane == 0) at = atomicAdd(rec.count, (unsigned long long)kBatch);
        at = __shfl_sync(FULL, at, 0);
        left = kBatch;
      }
      if (lane == 0 && at < rec.cap) {
        const uint64_t rows = reinterpret_cast<uint64_t>(L.base) + c0 * row_bytes<A>();
        rec.leaf[at] = make_uint4(uint32_t(rows), uint32_t(rows >> 32), m, had);
        rec.query[at] = query;
      }
      ++at;
      --left;
      had += uint32_t(__popc(m));
    }
    if (hit && lane == o) count = had;
  }
  // Room taken and not used is left as empty records.
  __device__ __forceinline__ void close(int lane) {
    for (uint32_t j = lane; j < left; j += 32)
      if (at + j < rec.cap) rec.leaf[at + j] = make_uint4(0, 0, 0, 0);
  }
};

template <typename A, int K, typename M, bool EXCL>
__global__ void __launch_bounds__(256) k_twithin_record(TreeView<A> tv0, Batch<A> b, A radius0,
                                                        uint64_t* __restrict__ counts,
                                                        HitRecords rec) {
  static_assert(RowLeaves<A, K>::value, "records name rows");
  extern __shared__ __align__(16) unsigned char tsmem[];
  A* slot = reinterpret_cast<A*>(tsmem) + threadIdx.x;
  const int stride = blockDim.x, lane = threadIdx.x & 31;
  TravStats st;
  CWithinRecord<A, K, M, EXCL> pol(rec);
  ThreadWalk<A, K, M> wk;
  coop_drive<A, K, M>(
      tv0, b, wk, pol, slot, stride, st,
      [&](uint64_t qi, const TreeView<A>&) {
        pol.radius = b.radius(radius0, qi);
        pol.count = 0;
        return true;
      },
      [&](int w, uint64_t qo) {
        const uint32_t cnt = shfl(pol.count, w);
        if (lane == 0) counts[qo] = cnt;
      });
  pol.close(lane);
}

// The records' hits at their queries' offsets.  A warp takes 32 records, a lane
// each: the record, then its query and offset, are one load for all of them;
// then the warp goes through the records kAhead at a time, lane p on the chunk's
// point p.  (A warp per four records, each lane loading the same record, waited
// on three dependent loads per four: 25M hits 506 us, 207 now.)
template <typename A, int K, typename M>
__global__ void __launch_bounds__(256) k_place_hits(const A* __restrict__ Q,
                                                    const uint64_t* __restrict__ offsets,
                                                    HitRecords rec, uint64_t n,
                                                    uint64_t capacity, A* __restrict__ out_d,
                                                    uint32_t* __restrict__ out_i) {
  constexpr int kAhead = 4;
  const int lane = threadIdx.x & 31;
  const uint64_t warps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  const unsigned below_me = (1u << lane) - 1u;
  for (uint64_t r0 = ((uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * 32; r0 < n;
       r0 += warps * 32) {
    uint4 mine = make_uint4(0, 0, 0, 0);
    uint64_t to = 0;
    A q[K];
#pragma unroll
    for (int d = 0; d < K; ++d) q[d] = A(0);
    if (r0 + lane < n) {
      mine = __ldg(rec.leaf + r0 + lane);
      if (mine.z) {
        const uint32_t query = __ldg(rec.query + r0 + lane);
        to = __ldg(offsets + query) + mine.w;
        // a row too short for its hits keeps the first of them
        const uint64_t end = min(__ldg(offsets + query + 1), capacity);
        while (mine.z && to + __popc(mine.z) > end) mine.z &= ~(0x80000000u >> __clz(mine.z));
#pragma unroll
        for (int d = 0; d < K; ++d) q[d] = __ldg(Q + uint64_t(query) * K + d);
      }
    }
    for (int j0 = 0; j0 < 32; j0 += kAhead) {
      A c[kAhead][K];
      uint32_t item[kAhead], mask[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        mask[j] = shfl(mine.z, j0 + j);
        const uint64_t rows = uint64_t(shfl(mine.y, j0 + j)) << 32 | shfl(mine.x, j0 + j);
        if ((mask[j] >> lane) & 1u)
          load_row<A, K>(reinterpret_cast<const uint8_t*>(rows), lane, c[j], item[j]);
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const uint64_t w = shfl64(to, j0 + j) + __popc(mask[j] & below_me);
        A oq[K];
#pragma unroll
        for (int d = 0; d < K; ++d) oq[d] = shfl(q[d], j0 + j);
        if ((mask[j] >> lane) & 1u) {
          out_d[w] = point_dist<M, A, K>(c[j], oq);
          out_i[w] = item[j];
        }
      }
    }
  }
}

template <typename A>
cudaError_t launch_within_record(const DeviceTree& t, const QueryLaunch& q, uint64_t* counts,
                                 const HitRecords& rec) {
  const TreeView<A> tv = make_view<A>(t);
  const Batch<A> b = make_batch<A>(q, kRefillCoop, kChunkRadius);
  return with_metric(q.metric, [&](auto m) {
    using M = decltype(m);
    return with_excl(q.exclusive, [&](auto ex) -> cudaError_t {
      constexpr bool EX = decltype(ex)::value;
      const size_t smem = size_t(t.max_stem_level + 2) * 256 * sizeof(A);
      auto kern = k_twithin_record<A, 3, M, EX>;
      const cudaError_t e =
          cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
      if (e != cudaSuccess) return e;
      kern<<<grid_for(kern, smem, (q.nq + 31) / 32), 256, smem, q.stream>>>(tv, b, A(q.radius),
                                                                            counts, rec);
      g_launches++;
      return cudaGetLastError();
    });
  });
}

template <typename A>
cudaError_t launch_place_hits(const QueryLaunch& q, const uint64_t* offsets, const HitRecords& rec,
                              uint64_t n) {
  if (n == 0) return cudaSuccess;
  return with_metric(q.metric, [&](auto m) {
    auto kern = k_place_hits<A, 3, decltype(m)>;
    kern<<<grid_for(kern, 0, (n + 31) / 32), 256, 0, q.stream>>>(
        static_cast<const A*>(q.queries), offsets, rec, n, q.capacity, static_cast<A*>(q.out_d),
        q.out_i);
    g_launches++;
    return cudaGetLastError();
  });
}

}  // namespace kgpu
