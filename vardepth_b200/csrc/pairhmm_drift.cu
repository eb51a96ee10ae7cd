// The drift tier (FP32, semiglobal): the pairs the primary tier spilled, because
// their likelihood lies more than 200 bits below a perfect match's (or, in a read of
// several strips, because a boundary did).
//
// A pair takes the long-read kernel's strips (pairhmm_long.cuh), one after another on
// one warp: every lane's state has its own power of two, chosen anew every 8 steps, so
// a path is kept however far it lies below the best one of its rows elsewhere in the
// haplotype.  (A boost per lane or per strip, held over the whole haplotype, follows
// the path that is best so far and drops the others: reads joined from two copies of a
// sequence came out up to 90 log10 too low, reads that hang off their haplotype up to
// 3 at a gap continuation of 0.1 and 46 at 0.005.)  Emission is two-sided, for the
// reads with Phred 0 and 1 bases.
//
// What goes on to FP64: reads of several strips that decay by more than long_max_bits,
// and every pair when the gap continuation is below kLongMinExt.
//
// The second half of the packed rows repeats the first: entries come in no order, and
// two that share a read rarely meet.
#include "pairhmm_launch.h"
#include "pairhmm_long.cuh"

namespace vd {
namespace {

template <int kBlocks>
__global__ void __launch_bounds__(kWarpsPerBlock * kWarp, kBlocks)
pairhmm_drift_kernel(const __grid_constant__ BatchView bv, const __grid_constant__ QueueView qv,
                     const Tables<float>* __restrict__ gtab, const __grid_constant__ Scalars<float> sc) {
  if (*qv.count == 0) return;
  __shared__ Tables<float> tab;
  __shared__ float4 rings[kWarpsPerBlock][2][kWarp];
  __shared__ int2 exps[kWarpsPerBlock][4];
  {
    const int words = (int)(sizeof(Tables<float>) / sizeof(int));
    const int* src = reinterpret_cast<const int*>(gtab);
    int* dst = reinterpret_cast<int*>(&tab);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & (kWarp - 1), wid = threadIdx.x >> 5;
  const long long gw = (long long)blockIdx.x * kWarpsPerBlock + wid;
  float4* const bufs = reinterpret_cast<float4*>(qv.scratch) + gw * qv.scratch_stride;
  const long long half = qv.scratch_stride / 2;
  long long total = qv.n_items;
  const long long c = (long long)*qv.count;
  total = c < total ? c : total;
  for (;;) {
    unsigned long long i = 0;
    if (lane == 0) i = atomicAdd(qv.head, 1ull);
    i = __shfl_sync(0xffffffffu, i, 0);
    if ((long long)i >= total) break;
    const RescueEntry e = qv.entries[i];
    WorkItem w;
    w.read = e.read;
    w.nhap = 1;
    w.hap_begin = e.hap;
    w.out_begin = e.out;
    w.code = bv.read_code[e.read];
    w.read2 = -1;
    w.out2_begin = 0;
    const int R = code_R(w.code);
    const int n = (int)(bv.read_off[e.read + 1] - bv.read_off[e.read]);
    const int nstrips = (n + kWarp * R - 1) / (kWarp * R);
    unsigned failed = sc.x < kLongMinExt ? 1u : 0u;
    for (int strip = 0; strip < nstrips && !(failed & 1u); ++strip) {
      switch (R) {
#define VD_DCASE(r)                                                                                               \
  case r:                                                                                                         \
    long_task<r, kLongSpanShort, true, true>(bv, qv, w, 0, strip, nstrips, 0, &tab, sc, lane, bufs, half, strip & 1, \
                                             rings[wid][0], rings[wid][1], exps[wid], failed);                    \
    break;
        VD_DCASE(1) VD_DCASE(2) VD_DCASE(3) VD_DCASE(4) VD_DCASE(5) VD_DCASE(6) VD_DCASE(7) VD_DCASE(8)
#undef VD_DCASE
        default: break;
      }
    }
    // (what fails in its last strip is handed on there; the output is NaN from the primary tier)
    if ((failed & 1u) && lane == 0) spill_pair<float>(qv, e.read, e.hap, e.out);
    __syncwarp();
  }
}

constexpr int kDriftBlocks = 3;

}  // namespace

cudaError_t launch_drift_f32(const BatchView& bv, const QueueView& qv, const Tables<float>* tab,
                             const Scalars<float>& sc, int grid, cudaStream_t stream) {
  pairhmm_drift_kernel<kDriftBlocks><<<grid, kWarpsPerBlock * kWarp, 0, stream>>>(bv, qv, tab, sc);
  return cudaGetLastError();
}

cudaError_t occupancy_drift_f32(int* blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, pairhmm_drift_kernel<kDriftBlocks>,
                                                       kWarpsPerBlock * kWarp, 0);
}

}  // namespace vd
