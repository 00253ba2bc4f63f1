// kernels_f64_hits.cu — one-walk radius kernels instantiated for double coordinates.
#include "kgpu_launch_impl.cuh"

#include "kgpu_hits.cuh"

namespace kgpu {
template cudaError_t launch_within_record<double>(const DeviceTree&, const QueryLaunch&, uint64_t*,
                                                  const HitRecords&);
template cudaError_t launch_place_hits<double>(const QueryLaunch&, const uint64_t*,
                                               const HitRecords&, uint64_t);
}  // namespace kgpu
