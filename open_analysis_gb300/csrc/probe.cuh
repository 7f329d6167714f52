// Probe samples, shared by the probe kernels (kernels.cu) and the direct sweeps (slab.cu).
#pragma once

#include "oafdtd_internal.cuh"

namespace oafdtd {

constexpr int kProbeLanes = 128;  // threads of a probe sum, whatever the block holds: one summation order

// Weighted float64 sum of probe pid for member b, in a fixed order; the whole block calls it, thread
// 0 has the result.
template <typename real>
__device__ __forceinline__ double probe_sum(const ProbeArgs<real>& a, int kind, int pid, int b) {
  __shared__ double warp_sum[kProbeLanes / 32];
  const int tid = (int)(threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z));
  const real* F = a.F[3 * kind + a.comp[pid]] + (long long)b * a.bs;
  double acc = 0.0;
  if (tid < kProbeLanes) {
#pragma unroll 1
    for (long long e = a.off[pid] + tid; e < a.off[pid + 1]; e += kProbeLanes)
      acc += (double)F[a.flat[e]] * a.w[e];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((tid & 31) == 0) warp_sum[tid >> 5] = acc;
  }
  __syncthreads();
  double s = 0.0;
  if (tid == 0)
    for (int w = 0; w < kProbeLanes / 32; ++w) s += warp_sum[w];
  __syncthreads();
  return s;
}

// The sample of one probe of one kind (0 E, 1 H) for one member (block = probe within the kind x
// members) at step step_base + off: kept for the running DFT of the chunk (vals) and in the recorded
// series.
template <typename real>
__device__ __forceinline__ void probe_sample(const ProbeArgs<real>& a, int kind, int block, int off) {
  const int pid = a.list[kind][block / a.B], b = block % a.B;
  const double s = probe_sum(a, kind, pid, b);
  if ((threadIdx.x | threadIdx.y | threadIdx.z) == 0) {
    const long long pb = (long long)pid * a.B + b;
    a.vals[pb * kChunk + off] = s;
    if (a.series != nullptr) a.series[pb * a.max_steps + *a.step_base + off] = s;
  }
}

}  // namespace oafdtd
