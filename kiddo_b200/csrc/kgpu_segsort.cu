// kgpu_segsort.cu — stable sort of every CSR segment by distance (the sorted
// radius families).
//
// A segment's entries are sorted as (distance, position) keys.  Keys are
// unique, so any sort of them is the stable sort of the distances, as
// Vec::sort; distances are +0 or more and never NaN (only hits are stored), so
// their bit patterns order like their values.  The items are gathered through
// the positions once the order is known.
//
//  * up to 8 hits: one lane's registers; 9..32: one warp's lanes
//    (k_seg_sort_small, which also lists the longer segments by class);
//  * 33..512: one warp, up to 16 keys per lane in registers; 513..4096: one
//    block of 128 threads, up to 32 keys per thread (k_seg_sort_mid);
//  * above: one block of 512 threads, 8192 (f64) or 16384 (f32) keys at a
//    time, and merges of such runs in global memory (k_seg_sort_long).
//
// What bounds it: instruction issue (a bitonic network of log2(n) stages on
// 64-bit keys); the hits cross HBM once each way.  Keys stay in registers, 8 to
// 32 independent compare-exchanges per thread and step, so no step waits on a
// dependent load; shared memory only carries the strides between warps, two
// passes per power of two above a warp's run.  The merge sort in shared memory
// that this replaced (one dependent load per merged entry, 16 warps per SM)
// took 15.8 ms for the 87M hits of 1M radius queries over 32 catalogues (2.5 ms
// now), and 3.4 ms for the 25M hits of 1M cross-match queries (0.55 ms now).
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "kgpu_bitonic.cuh"
#include "kgpu_devbuf.h"
#include "kgpu_device.cuh"
#include "kgpu_launch.h"

namespace kgpu {

namespace {

// Stable sort of the n <= T * E entries at (d, it) by T threads (a warp of its
// own slice of shared memory when T == 32, else the whole block).
template <typename A, int T, int E>
__device__ __forceinline__ void sort_run(A* __restrict__ d, uint32_t* __restrict__ it, uint32_t n,
                                         unsigned char* smem, int tid) {
  using Key = KeyOf<A>;
  KeyStore<Key> sm = KeyStore<Key>::at(smem, T * E);
  auto sync = [] {
    if constexpr (T == 32) __syncwarp();
    else __syncthreads();
  };
  Key k[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const uint32_t i = uint32_t(e) * T + tid;
    k[e] = i < n ? Key::make(d[i], i) : Key::last();
  }
  warp_sort<Key, E>(k, tid & 31);
  if constexpr (T > 32) block_merges<Key, T, E, 64 * E>(k, sm, tid);
  // back to coalesced order; every item is read before any is overwritten
  sync();
#pragma unroll
  for (int e = 0; e < E; ++e) sm.put(uint32_t(tid) * E + e, k[e]);
  sync();
  uint32_t v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const uint32_t i = uint32_t(e) * T + tid;
    v[e] = 0;
    if (i < n) v[e] = it[sm.get(i).pos()];
  }
  sync();
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const uint32_t i = uint32_t(e) * T + tid;
    if (i < n) {
      d[i] = sm.get(i).dist();
      it[i] = v[e];
    }
  }
  sync();
}

// ---- segment lists --------------------------------------------------------------
// Longer segments by the size their sort pads to: 64, 128, ... 4096, then all
// above (class 7).  Each class has its own list of segment numbers.
constexpr int kClasses = 8;
__host__ __device__ inline int class_of(uint64_t n) {  // n >= 33
  int c = 0;
  while (c < kClasses - 1 && n > (uint64_t(64) << c)) ++c;
  return c;
}
struct SegLists {
  uint32_t* seg[kClasses];           // segment numbers
  unsigned long long* count;         // [kClasses] entries
  unsigned long long* taken;         // [kClasses] entries handed out
};

// Stable sort of one segment of n <= N hits by its own thread: the segment is
// loaded into registers (padding +inf after it), insertion-sorted by a fully
// unrolled network of adjacent compare-swaps that swap only strictly greater
// keys (so equal keys keep their order and padding stays behind), and written
// back.
template <typename A, int N>
__device__ __forceinline__ void small_segment_sort(A* __restrict__ d, uint32_t* __restrict__ it,
                                                   uint32_t n) {
  A kd[N];
  uint32_t kv[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    kd[j] = uint32_t(j) < n ? d[j] : inf_of<A>();
    kv[j] = uint32_t(j) < n ? it[j] : 0u;
  }
#pragma unroll
  for (int a = 1; a < N; ++a) {
#pragma unroll
    for (int j = a; j > 0; --j) {
      const bool sw = kd[j - 1] > kd[j];
      const A td = kd[j - 1];
      const uint32_t tv = kv[j - 1];
      kd[j - 1] = sw ? kd[j] : td;
      kv[j - 1] = sw ? kv[j] : tv;
      kd[j] = sw ? td : kd[j];
      kv[j] = sw ? tv : kv[j];
    }
  }
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (uint32_t(j) < n) {
      d[j] = kd[j];
      it[j] = kv[j];
    }
}

// Segments of up to 32 hits.  A warp takes 32 segments at a time (lane l
// reads segment base + l's bounds, coalesced): segments of 2..kThreadSort
// hits are sorted in registers by their own lane (small_segment_sort), the
// warp sorts its segments of kThreadSort+1..32 hits one after another, one key
// per lane, and longer segments go on their class's list.
template <typename A>
__global__ void __launch_bounds__(256) k_seg_sort_small(const uint64_t* __restrict__ offsets,
                                                        uint64_t nq, uint64_t capacity,
                                                        A* __restrict__ d,
                                                        uint32_t* __restrict__ it,
                                                        SegLists lists) {
  constexpr uint64_t kThreadSort = 8;
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t base = warp * 32; base < nq; base += nwarps * 32) {
    const uint64_t s = base + lane;
    uint64_t o = 0, n = 0;
    if (s < nq) {
      o = min(offsets[s], capacity);
      n = max(min(offsets[s + 1], capacity), o) - o;
    }
    if (n >= 2 && n <= 4) {
      small_segment_sort<A, 4>(d + o, it + o, uint32_t(n));
    } else if (n > 4 && n <= kThreadSort) {
      small_segment_sort<A, kThreadSort>(d + o, it + o, uint32_t(n));
    }
    for (unsigned big = __ballot_sync(FULL, n > kThreadSort && n <= 32); big; big &= big - 1) {
      const int src = __ffs(big) - 1;
      const uint64_t so = __shfl_sync(FULL, (unsigned long long)o, src);
      const uint32_t sn = uint32_t(__shfl_sync(FULL, (unsigned long long)n, src));
      KeyOf<A> k[1];
      uint32_t v = 0;
      k[0] = KeyOf<A>::last();
      if (uint32_t(lane) < sn) {
        k[0] = KeyOf<A>::make(d[so + lane], lane);
        v = it[so + lane];
      }
      warp_sort<KeyOf<A>, 1>(k, lane);
      v = __shfl_sync(FULL, v, int(k[0].pos() & 31u));
      if (uint32_t(lane) < sn) {
        d[so + lane] = k[0].dist();
        it[so + lane] = v;
      }
    }
    if (__any_sync(FULL, n > 32)) {
      const int c = n > 32 ? class_of(n) : -1;
      for (int j = 0; j < kClasses; ++j) {
        const unsigned m = __ballot_sync(FULL, c == j);
        if (!m) continue;
        const int lead = __ffs(m) - 1;
        unsigned long long at = 0;
        if (lane == lead) at = atomicAdd(lists.count + j, (unsigned long long)__popc(m));
        at = __shfl_sync(FULL, at, lead);
        if (c == j) lists.seg[j][at + __popc(m & ((1u << lane) - 1u))] = uint32_t(s);
      }
    }
  }
}

// Segments of 33..4096 hits, longest first: a block of 128 threads per segment
// above 512, then a warp per segment.  Four blocks per SM in f32 (128
// registers), three in f64 (168), where 32 keys per thread take 96.
template <typename A>
__global__ void __launch_bounds__(128, sizeof(A) == 4 ? 4 : 3) k_seg_sort_mid(const uint64_t* __restrict__ offsets,
                                                      uint64_t capacity, A* __restrict__ d,
                                                      uint32_t* __restrict__ it, SegLists lists) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long next;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int c = 6; c >= 4; --c) {  // 4096, 2048, 1024
    const unsigned long long cnt = lists.count[c];
    for (;;) {
      __syncthreads();
      if (tid == 0) next = atomicAdd(lists.taken + c, 1ull);
      __syncthreads();
      const unsigned long long j = next;
      if (j >= cnt) break;
      const uint32_t s = lists.seg[c][j];
      const uint64_t o = min(offsets[s], capacity);
      const uint32_t n = uint32_t(min(offsets[s + 1], capacity) - o);
      if (c == 6) sort_run<A, 128, 32>(d + o, it + o, n, smem, tid);
      else if (c == 5) sort_run<A, 128, 16>(d + o, it + o, n, smem, tid);
      else sort_run<A, 128, 8>(d + o, it + o, n, smem, tid);
    }
  }
  __syncthreads();
  unsigned char* mine = smem + (tid >> 5) * KeyStore<KeyOf<A>>::bytes(512);
  for (int c = 3; c >= 0; --c) {  // 512, 256, 128, 64
    const unsigned long long cnt = lists.count[c];
    for (;;) {
      unsigned long long j = 0;
      if (lane == 0) j = atomicAdd(lists.taken + c, 1ull);
      j = __shfl_sync(FULL, j, 0);
      if (j >= cnt) break;
      const uint32_t s = lists.seg[c][j];
      const uint64_t o = min(offsets[s], capacity);
      const uint32_t n = uint32_t(min(offsets[s + 1], capacity) - o);
      if (c == 3) sort_run<A, 32, 16>(d + o, it + o, n, mine, lane);
      else if (c == 2) sort_run<A, 32, 8>(d + o, it + o, n, mine, lane);
      else if (c == 1) sort_run<A, 32, 4>(d + o, it + o, n, mine, lane);
      else sort_run<A, 32, 2>(d + o, it + o, n, mine, lane);
    }
  }
}

// Stable merge step (merge path): out[lo..hi) from runs a[0..na) and b[0..nb),
// ties taken from `a` first.
template <typename A>
__device__ __forceinline__ void merge_range(const A* ad, const uint32_t* ai, uint32_t na,
                                            const A* bd, const uint32_t* bi, uint32_t nb,
                                            A* od, uint32_t* oi, uint32_t lo, uint32_t hi) {
  if (lo >= hi) return;
  uint32_t l = lo > nb ? lo - nb : 0, h = lo < na ? lo : na;
  while (l < h) {
    const uint32_t mid = (l + h) >> 1;
    if (!(bd[lo - mid - 1] < ad[mid])) l = mid + 1;  // ad[mid] <= bd[...]: a first
    else h = mid;
  }
  uint32_t x = l, y = lo - l;
  for (uint32_t o = lo; o < hi; ++o) {
    bool take_a = x < na && (y >= nb || !(bd[y] < ad[x]));
    if (take_a) { od[o] = ad[x]; oi[o] = ai[x]; ++x; }
    else { od[o] = bd[y]; oi[o] = bi[y]; ++y; }
  }
}

// Merges the sorted runs of `width` entries of one segment until one is left,
// by the whole block, ping-ponging between (d0, i0) and (d1, i1).  Returns true
// if the result ended in (d1, i1).
template <typename A>
__device__ bool block_merge_runs(A* d0, uint32_t* i0, A* d1, uint32_t* i1, uint32_t n,
                                 uint32_t width) {
  bool in1 = false;
  for (; width < n; width <<= 1) {
    A* sd = in1 ? d1 : d0;
    uint32_t* si = in1 ? i1 : i0;
    A* td = in1 ? d0 : d1;
    uint32_t* ti = in1 ? i0 : i1;
    const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
    const uint32_t lo = threadIdx.x * per;
    const uint32_t hi = min(n, lo + per);
    // each thread's output range may span several run pairs
    uint32_t o = lo;
    while (o < hi) {
      const uint32_t pair = o / (2 * width);
      const uint32_t start = pair * 2 * width;
      const uint32_t mid = min(n, start + width);
      const uint32_t end = min(n, start + 2 * width);
      const uint32_t stop = min(hi, end);
      merge_range<A>(sd + start, si + start, mid - start, sd + mid, si + mid, end - mid,
                     td + start, ti + start, o - start, stop - start);
      o = stop;
    }
    __syncthreads();
    in1 = !in1;
  }
  return in1;
}

// Segments above 4096 hits, a block each: in runs of up to kRun entries, which
// are then merged in global memory with `scratch` as the second buffer.
template <typename A>
__global__ void __launch_bounds__(512) k_seg_sort_long(const uint64_t* __restrict__ offsets,
                                                       uint64_t capacity, A* __restrict__ d,
                                                       uint32_t* __restrict__ it,
                                                       A* __restrict__ scratch_d,
                                                       uint32_t* __restrict__ scratch_i,
                                                       SegLists lists) {
  constexpr uint32_t kRun = sizeof(A) == 4 ? 16384 : 8192;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long next;
  const int tid = threadIdx.x;
  const unsigned long long cnt = lists.count[kClasses - 1];
  for (;;) {
    __syncthreads();
    if (tid == 0) next = atomicAdd(lists.taken + kClasses - 1, 1ull);
    __syncthreads();
    const unsigned long long j = next;
    if (j >= cnt) break;
    const uint32_t s = lists.seg[kClasses - 1][j];
    const uint64_t o = min(offsets[s], capacity);
    const uint32_t n = uint32_t(min(offsets[s + 1], capacity) - o);
    for (uint32_t r = 0; r < n; r += kRun) {
      const uint32_t m = min(kRun, n - r);
      if (m <= 8192) {
        sort_run<A, 512, 16>(d + o + r, it + o + r, m, smem, tid);
      } else {
        if constexpr (sizeof(A) == 4) sort_run<A, 512, 32>(d + o + r, it + o + r, m, smem, tid);
      }
    }
    if (n > kRun && block_merge_runs<A>(d + o, it + o, scratch_d + o, scratch_i + o, n, kRun)) {
      for (uint32_t x = tid; x < n; x += blockDim.x) {
        d[o + x] = scratch_d[o + x];
        it[o + x] = scratch_i[o + x];
      }
      __syncthreads();
    }
  }
}

template <typename Kern>
int blocks_per_sm(Kern kern, int threads, size_t smem) {
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, threads, smem) != cudaSuccess || b < 1)
    b = 1;
  return b;
}

}  // namespace

template <typename A>
cudaError_t launch_seg_sort(const uint64_t* offsets, uint64_t nq, uint64_t capacity, A* d,
                            uint32_t* it, A* scratch_d, uint32_t* scratch_i, cudaStream_t s) {
  if (nq == 0) return cudaSuccess;
  using Key = KeyOf<A>;
  // class c holds segments above 32 << c (33, 65, ... 4097 hits and more), so
  // its list has at most capacity / that many entries
  SegLists lists;
  uint64_t room[kClasses], total = 0;
  for (int c = 0; c < kClasses; ++c) {
    room[c] = std::min<uint64_t>(nq, capacity / ((uint64_t(32) << c) + 1) + 1);
    total += room[c];
  }
  DevBuf buf;
  const size_t counters = 2 * kClasses * sizeof(unsigned long long);
  cudaError_t e = buf.alloc(counters + total * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(buf.p, 0, counters, s);
  if (e != cudaSuccess) return e;
  lists.count = buf.as<unsigned long long>();
  lists.taken = lists.count + kClasses;
  uint32_t* seg = reinterpret_cast<uint32_t*>(lists.taken + kClasses);
  for (int c = 0; c < kClasses; ++c) {
    lists.seg[c] = seg;
    seg += room[c];
  }
  const int sms = sm_count();
  {
    auto kern = k_seg_sort_small<A>;
    const uint64_t full = uint64_t(blocks_per_sm(kern, 256, 0)) * sms;
    const uint64_t need = (nq + 255) / 256;
    kern<<<unsigned(std::min(need, full)), 256, 0, s>>>(offsets, nq, capacity, d, it, lists);
    g_launches++;
  }
  if (capacity > 4096) {
    auto kern = k_seg_sort_long<A>;
    const size_t smem = KeyStore<Key>::bytes(sizeof(A) == 4 ? 16384 : 8192);
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem))) !=
        cudaSuccess)
      return e;
    const uint64_t full = uint64_t(blocks_per_sm(kern, 512, smem)) * sms;
    kern<<<unsigned(std::min(room[kClasses - 1], full)), 512, smem, s>>>(
        offsets, capacity, d, it, scratch_d, scratch_i, lists);
    g_launches++;
  }
  if (capacity > 32) {
    auto kern = k_seg_sort_mid<A>;
    const size_t smem = std::max(KeyStore<Key>::bytes(4096), 4 * KeyStore<Key>::bytes(512));
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem))) !=
        cudaSuccess)
      return e;
    const uint64_t full = uint64_t(blocks_per_sm(kern, 128, smem)) * sms;
    kern<<<unsigned(std::min((room[0] + 3) / 4 + room[4], full)), 128, smem, s>>>(
        offsets, capacity, d, it, lists);
    g_launches++;
  }
  return cudaGetLastError();
}
template cudaError_t launch_seg_sort<float>(const uint64_t*, uint64_t, uint64_t, float*, uint32_t*,
                                            float*, uint32_t*, cudaStream_t);
template cudaError_t launch_seg_sort<double>(const uint64_t*, uint64_t, uint64_t, double*,
                                             uint32_t*, double*, uint32_t*, cudaStream_t);

}  // namespace kgpu
