// kgpu_hits.h — what a counting pass keeps for the filling pass (kgpu_hits).
#pragma once

#include <cstdint>

#include "kgpu_devbuf.h"
#include "kgpu_launch.h"

// The processing order and, where the counting pass recorded them, the places
// of a batch's hits; all on the stream of the counting call.
struct kgpu_hits {
  const void* owner = nullptr;  // the tree or forest counted; its leaves are what `rec` names
  kgpu::DevBuf order, order_tmp, counters;
  // The records, which a fill short of scratch gives up (it then walks again).  They
  // are not given up before, useful or not: blocks freed between the two calls
  // leave the pool's free ranges in pieces, and the sort's scratch then waits for
  // memory to be mapped again (90M hits 9.9 ms a call, 10 to 84 now and then).
  mutable kgpu::DevBuf leaf, query;
  kgpu::HitRecords rec;
  bool ordered = false;
  mutable uint64_t recorded = ~uint64_t(0);  // records to place; ~0: none are kept
  uint64_t nq = 0, total = 0;

  void drop_records() const {
    for (kgpu::DevBuf* b : {&leaf, &query}) {
      if (b->p) cudaFreeAsync(b->p, b->s);
      b->p = nullptr;
    }
    recorded = ~uint64_t(0);
  }
};

namespace kgpu {
// Counts every query's hits, scans them into offsets[0..nq] and keeps what the
// fill needs; `q` describes the batch (order included in `hits`).  Waits for
// the total.  Returns a kgpu_status.
int radius_count_keep(const DeviceTree& dt, QueryLaunch& q, uint64_t* offsets, kgpu_hits& hits);
// Writes and (q.sorted) sorts the hits.
int radius_fill_kept(const DeviceTree& dt, QueryLaunch& q, const uint64_t* offsets,
                     const kgpu_hits& hits);
}  // namespace kgpu
