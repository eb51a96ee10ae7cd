// Instantiations of the long-read kernel (pairhmm_long.cuh): strips of up to
// 256 rows (5-8 rows per lane) and of 128 rows (4 rows per lane).
#include "pairhmm_launch.h"
#include "pairhmm_long.cuh"

namespace vd {

cudaError_t launch_long_f32(int R, const BatchView& bv, const QueueView& qv, const Tables<float>* tab,
                            const Scalars<float>& sc, int grid, cudaStream_t stream) {
  const int threads = kWarpsPerBlock * kWarp;
  // (gap continuations below 0.08 choose the lanes' exponents twice as often)
  if (sc.x >= 0.08f) {
    if (R == 8) pairhmm_long_kernel<5, 8, 3, kLongSpan><<<grid, threads, 0, stream>>>(bv, qv, tab, sc);
    else pairhmm_long_kernel<4, 4, 4, kLongSpan><<<grid, threads, 0, stream>>>(bv, qv, tab, sc);
  } else {
    if (R == 8) pairhmm_long_kernel<5, 8, 3, kLongSpanShort><<<grid, threads, 0, stream>>>(bv, qv, tab, sc);
    else pairhmm_long_kernel<4, 4, 4, kLongSpanShort><<<grid, threads, 0, stream>>>(bv, qv, tab, sc);
  }
  return cudaGetLastError();
}

cudaError_t occupancy_long_f32(int R, int* blocks_per_sm) {
  const int threads = kWarpsPerBlock * kWarp;
  return R == 8 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, pairhmm_long_kernel<5, 8, 3, kLongSpan>, threads, 0)
                : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, pairhmm_long_kernel<4, 4, 4, kLongSpan>, threads, 0);
}

}  // namespace vd
