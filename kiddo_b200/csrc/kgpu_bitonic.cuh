// kgpu_bitonic.cuh — sorting networks over keys held in registers.
//
// A Key has operator< (a strict order; equal keys may change places),
// from_lane(mask) (the key of lane ^ mask) and a KeyStore specialisation.
#pragma once

#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "kgpu_device.cuh"

namespace kgpu {

// N keys in shared memory, one pad slot after every 16, so that threads 8, 16
// or 32 entries apart touch different banks.
template <typename Key>
struct KeyStore;

// Words below kLastWord, the largest finite double, order like the doubles with
// their bits (denormals included), and one comparison of those takes the place of
// two on the halves, on a pipe that is idle here: the moves of a
// compare-exchange keep the other one busy.
constexpr unsigned long long kLastWord = 0x7fefffffffffffffull;
__device__ __forceinline__ bool word_less(unsigned long long a, unsigned long long b) {
  return __longlong_as_double((long long)a) < __longlong_as_double((long long)b);
}

// Distances with a place: unique keys, so any sort of them is a stable sort of
// the distances.  Distances are +0 or more and never NaN, so their bit patterns
// order like their values.
// f32: distance bits above the position in one 64-bit word.  f64: the distance
// and the position.
struct KeyF32 {
  unsigned long long v;
  __device__ __forceinline__ static KeyF32 make(float d, uint32_t p) {
    return {(static_cast<unsigned long long>(__float_as_uint(d)) << 32) | p};
  }
  __device__ __forceinline__ static KeyF32 last() { return {kLastWord}; }
  __device__ __forceinline__ bool operator<(const KeyF32& o) const { return word_less(v, o.v); }
  __device__ __forceinline__ float dist() const { return __uint_as_float(uint32_t(v >> 32)); }
  __device__ __forceinline__ uint32_t pos() const { return uint32_t(v); }
  __device__ __forceinline__ KeyF32 from_lane(int mask) const {
    return {__shfl_xor_sync(FULL, v, mask)};
  }
};
struct KeyF64 {
  double d;
  uint32_t p;
  __device__ __forceinline__ static KeyF64 make(double d, uint32_t p) { return {d, p}; }
  __device__ __forceinline__ static KeyF64 last() { return {inf_of<double>(), ~0u}; }
  // three chained comparisons, against six or so on the words of the two numbers
  __device__ __forceinline__ bool operator<(const KeyF64& o) const {
    return d < o.d || (d == o.d && p < o.p);
  }
  __device__ __forceinline__ double dist() const { return d; }
  __device__ __forceinline__ uint32_t pos() const { return p; }
  __device__ __forceinline__ KeyF64 from_lane(int mask) const {
    return {__shfl_xor_sync(FULL, d, mask), __shfl_xor_sync(FULL, p, mask)};
  }
};
template <typename A>
using KeyOf = typename std::conditional<sizeof(A) == 4, KeyF32, KeyF64>::type;

// in shared memory, one pad slot after every 16
template <>
struct KeyStore<KeyF32> {
  unsigned long long* v;
  __host__ __device__ static constexpr size_t slots(uint32_t n) { return n + n / 16; }
  __host__ __device__ static constexpr size_t bytes(uint32_t n) { return slots(n) * 8; }
  __device__ static KeyStore at(unsigned char* p, uint32_t) {
    return {reinterpret_cast<unsigned long long*>(p)};
  }
  __device__ __forceinline__ KeyF32 get(uint32_t i) const { return {v[i + (i >> 4)]}; }
  __device__ __forceinline__ void put(uint32_t i, const KeyF32& k) { v[i + (i >> 4)] = k.v; }
};
template <>
struct KeyStore<KeyF64> {
  double* v;
  uint32_t* p;
  __host__ __device__ static constexpr size_t slots(uint32_t n) { return n + n / 16; }
  __host__ __device__ static constexpr size_t bytes(uint32_t n) { return slots(n) * 12; }
  __device__ static KeyStore at(unsigned char* m, uint32_t n) {
    double* v = reinterpret_cast<double*>(m);
    return {v, reinterpret_cast<uint32_t*>(v + slots(n))};
  }
  __device__ __forceinline__ KeyF64 get(uint32_t i) const {
    return {v[i + (i >> 4)], p[i + (i >> 4)]};
  }
  __device__ __forceinline__ void put(uint32_t i, const KeyF64& k) {
    v[i + (i >> 4)] = k.d;
    p[i + (i >> 4)] = k.p;
  }
};

// All comparators ascend (the lower index keeps the smaller key): the first
// step of each power of two pairs index i with its mirror in the block, the
// later steps pair i with i ^ stride.
template <typename Key>
__device__ __forceinline__ void order_pair(Key& a, Key& b) {
  const bool sw = b < a;
  const Key t = a;
  a = sw ? b : a;
  b = sw ? t : b;
}

// Strides STRIDE, STRIDE / 2, ... 1 over a warp's 32 * E keys held blocked
// (lane t has indices t * E + e).
template <typename Key, int E, int STRIDE>
__device__ __forceinline__ void warp_strides(Key (&k)[E], int lane) {
  if constexpr (STRIDE >= E) {
    constexpr int M = STRIDE / E;
    const bool low = (lane & M) == 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const Key o = k[e].from_lane(M);
      k[e] = ((o < k[e]) == low) ? o : k[e];
    }
    if constexpr (STRIDE > 1) warp_strides<Key, E, STRIDE / 2>(k, lane);
  } else if constexpr (STRIDE >= 1) {
#pragma unroll
    for (int e = 0; e < E; ++e)
      if ((e & STRIDE) == 0) order_pair(k[e], k[e + STRIDE]);
    if constexpr (STRIDE > 1) warp_strides<Key, E, STRIDE / 2>(k, lane);
  }
}

// Sorts the warp's 32 * E keys: sizes SIZE, 2 SIZE, ... 32 E, or up to `limit`
// (a power of two, the same in every thread): runs of that many keys.
template <typename Key, int E, int SIZE = 2>
__device__ __forceinline__ void warp_sort(Key (&k)[E], int lane, int limit = 32 * E) {
  if constexpr (SIZE <= 32 * E) {
    if (SIZE > limit) return;
    if constexpr (SIZE <= E) {
#pragma unroll
      for (int e = 0; e < E; ++e)
        if ((e & (SIZE / 2)) == 0) order_pair(k[e], k[e ^ (SIZE - 1)]);
    } else {
      constexpr int M = SIZE / E - 1;
      const bool low = (lane & (SIZE / E / 2)) == 0;
      if constexpr (E == 1) {
        const Key o = k[0].from_lane(M);
        k[0] = ((o < k[0]) == low) ? o : k[0];
      } else {
#pragma unroll
        for (int e = 0; e < E / 2; ++e) {
          const Key a = k[E - 1 - e].from_lane(M), b = k[e].from_lane(M);
          k[e] = ((a < k[e]) == low) ? a : k[e];
          k[E - 1 - e] = ((b < k[E - 1 - e]) == low) ? b : k[E - 1 - e];
        }
      }
    }
    if constexpr (SIZE > 2) warp_strides<Key, E, SIZE / 4>(k, lane);
    warp_sort<Key, E, SIZE * 2>(k, lane, limit);
  }
}

// In-thread strides of keys held strided (thread t has indices e * T + t):
// index strides ES * T, ... T.
template <typename Key, int E, int ES>
__device__ __forceinline__ void thread_strides(Key (&k)[E]) {
  if constexpr (ES >= 1) {
#pragma unroll
    for (int e = 0; e < E; ++e)
      if ((e & ES) == 0) order_pair(k[e], k[e + ES]);
    thread_strides<Key, E, ES / 2>(k);
  }
}

// Sizes SIZE, 2 SIZE, ... T * E of a block of T threads whose warps hold
// sorted runs of SIZE / 2 keys, blocked in and blocked out.  Between warps the
// keys go through shared memory: written with the upper half of every
// SIZE-block mirrored (which turns the mirrored first step into a plain
// stride), read strided for the strides from SIZE / 2 down to T, and written
// back for the strides inside a warp.  Needs 32 * E >= T.  `limit` as above.
template <typename Key, int T, int E, int SIZE>
__device__ __forceinline__ void block_merges(Key (&k)[E], KeyStore<Key>& sm, int tid,
                                             int limit = T * E) {
  static_assert(32 * E >= T, "a warp's run must reach the strided strides");
  if constexpr (SIZE <= T * E) {
    if (SIZE > limit) return;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint32_t i = uint32_t(tid) * E + e;
      sm.put((i & (SIZE / 2)) ? i ^ (SIZE / 2 - 1) : i, k[e]);
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) k[e] = sm.get(uint32_t(e) * T + tid);
    thread_strides<Key, E, SIZE / 2 / T>(k);
    // each thread rewrites the slots that it read
#pragma unroll
    for (int e = 0; e < E; ++e) sm.put(uint32_t(e) * T + tid, k[e]);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) k[e] = sm.get(uint32_t(tid) * E + e);
    warp_strides<Key, E, (T / 2 < 16 * E ? T / 2 : 16 * E)>(k, tid & 31);
    block_merges<Key, T, E, SIZE * 2>(k, sm, tid, limit);
  }
}

}  // namespace kgpu
