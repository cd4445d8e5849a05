// The decode kernel at precision 1.
#include "nz_decode_kernel.cuh"

namespace nz {
template int launch_decode_precision<1>(int, const BatchArgs &, uint32_t, uint32_t, cudaStream_t);
}  // namespace nz
