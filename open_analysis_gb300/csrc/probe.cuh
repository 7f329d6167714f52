// Probe samples, shared by the probe kernels (kernels.cu) and the direct sweeps (slab.cu).
#pragma once

#include "oafdtd_internal.cuh"

namespace oafdtd {

constexpr int kProbeLanes = 128;  // threads of a probe sum, whatever the block holds: one summation order
// Terms of a lane loaded ahead of their additions: a probe is bound by the latency of its gathers. us a
// step of 200x160x80 with eight E and H probes of 11932 points, one / 8 / 16 ahead: 209 / 127.5 / 127; four
// of 107388 points: 1327 / 440 / 324 (126 and 125 with port probes alone). Registers as without.
constexpr int kProbeDepth = 16;

// Weighted float64 sum of probe pid for member b, in a fixed order; the whole block calls it, thread
// 0 has the result.
template <typename real>
__device__ __forceinline__ double probe_sum(const ProbeArgs<real>& a, int kind, int pid, int b) {
  __shared__ double warp_sum[kProbeLanes / 32];
  const int tid = (int)(threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z));
  const real* F = a.F[3 * kind + a.comp[pid]] + (long long)b * a.bs;
  double acc = 0.0;
  if (tid < kProbeLanes) {
    const long long end = a.off[pid + 1];
    long long e = a.off[pid] + tid;
#pragma unroll 1
    for (; e + (kProbeDepth - 1) * kProbeLanes < end; e += kProbeDepth * kProbeLanes) {
      double t[kProbeDepth];
#pragma unroll
      for (int u = 0; u < kProbeDepth; ++u) t[u] = (double)F[a.flat[e + u * kProbeLanes]] * a.w[e + u * kProbeLanes];
#pragma unroll
      for (int u = 0; u < kProbeDepth; ++u) acc += t[u];
    }
#pragma unroll 1
    for (; e < end; e += kProbeLanes) acc += (double)F[a.flat[e]] * a.w[e];
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
