// The decode kernel at precision 7.
#include "nz_decode_kernel.cuh"

namespace nz {
template int launch_decode_precision<7>(int, const BatchArgs &, uint32_t, uint32_t, cudaStream_t);
int launch_decode_exponents(const BatchArgs &b, uint32_t warps, uint32_t smem_bytes, cudaStream_t st) {
  return launch_decode<7, false>(b, warps, smem_bytes, st);
}
}  // namespace nz
