// Kernels of the learned S-parameter surrogate: a BF16 tensor-core GEMM with FP32 accumulation
// and fused epilogues (bias, ReLU or tanh, and their derivatives), the loss gradient, bias gradients and
// the Adam update. The surrogate's training loop (open_analysis_gb300/surrogate.py) drives them
// on device buffers it owns; nothing here allocates.
//
// GEMM: C (M x N) = op(A) (M x K) . op(B) (K x N), op = identity or transpose per the flags:
//   A: row-major M x K (ta = 0) or row-major K x M (ta = 1), leading dimension lda;
//   B: row-major K x N (tb = 0) or row-major N x K (tb = 1), leading dimension ldb.
// Main path (gemm_pipe_kernel): a block computes a BM x 64 tile (BM = 64, or 32 when 64-row tiles
// would leave most of the SMs idle) with 4 warps (2 x 2) as 16 x 8 x 16 warp MMAs (mma.sync
// m16n8k16, BF16 in, FP32 accumulate). K advances 32 at a time through a 3-stage shared-memory
// ring filled by 16-byte cp.async copies, each operand tile stored as it lies in global memory
// (K-contiguous or M/N-contiguous); ldmatrix (.trans for the M/N-contiguous layouts) turns it into
// MMA fragments. Needs M, N, K, lda, ldb multiples of 8 and 16-byte aligned operands.
// Fallback (gemm_bf16_kernel): scalar staging, any sizes and alignments, for ragged shapes.

#include <cuda_bf16.h>
#include <stdint.h>

#include <cstring>

#include "../../include/oafdtd.h"
#include "oafdtd_internal.cuh"

namespace oafdtd {

constexpr int kBM = 64, kBN = 64, kBK = 32, kPadK = kBK + 8;  // +8 BF16: rows 80 bytes apart

struct GemmArgs {
  const __nv_bfloat16* A;
  const __nv_bfloat16* B;
  float* C32;             // FP32 result (nullable)
  __nv_bfloat16* C16;     // BF16 result (nullable)
  const float* bias;      // per column (nullable)
  const __nv_bfloat16* mask;  // activations for epilogues 2 and 4, same layout as C (nullable)
  // act: 0 none, 1 ReLU, 2 keep where mask > 0 (ReLU derivative), 3 tanh, 4 multiply by
  // 1 - mask^2 (tanh derivative, mask = the stored tanh output)
  int M, N, K, lda, ldb, ldc, ta, tb, act;
  float beta;             // C32 = acc + beta * C32 (gradient accumulation); 0 overwrites
  long long sA, sB, sC, sBias;  // elements between groups (blockIdx.z); the mask moves with C
};

// The arguments of group blockIdx.z.
__device__ __forceinline__ GemmArgs at_group(const GemmArgs& g0) {
  GemmArgs g = g0;
  const long long z = blockIdx.z;
  if (z) {
    g.A += z * g.sA;
    g.B += z * g.sB;
    if (g.C32) g.C32 += z * g.sC;
    if (g.C16) g.C16 += z * g.sC;
    if (g.mask) g.mask += z * g.sC;
    if (g.bias) g.bias += z * g.sBias;
  }
  return g;
}

__device__ __forceinline__ uint32_t pack2(const __nv_bfloat16* p) {
  return *reinterpret_cast<const uint32_t*>(p);
}

__global__ void __launch_bounds__(128) gemm_bf16_kernel(const GemmArgs g0) {
  const GemmArgs g = at_group(g0);
  __shared__ __align__(16) __nv_bfloat16 As[kBM][kPadK];
  __shared__ __align__(16) __nv_bfloat16 Bs[kBN][kPadK];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int grp = lane >> 2, tig = lane & 3;
  float acc[2][4][4] = {};
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  for (int k0 = 0; k0 < g.K; k0 += kBK) {
    // stage A (rows m, k contiguous) and B (columns n, k contiguous)
    for (int e = tid; e < kBM * kBK; e += blockDim.x) {
      const int r = e / kBK, kk = e % kBK;
      const int m = m0 + r, k = k0 + kk;
      __nv_bfloat16 v = zero;
      if (m < g.M && k < g.K) v = g.ta ? g.A[(long long)k * g.lda + m] : g.A[(long long)m * g.lda + k];
      As[r][kk] = v;
    }
    for (int e = tid; e < kBN * kBK; e += blockDim.x) {
      const int c = e / kBK, kk = e % kBK;
      const int n = n0 + c, k = k0 + kk;
      __nv_bfloat16 v = zero;
      if (n < g.N && k < g.K) v = g.tb ? g.B[(long long)n * g.ldb + k] : g.B[(long long)k * g.ldb + n];
      Bs[c][kk] = v;
    }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < kBK; ks += 16) {
      uint32_t a[2][4], b[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm + 16 * i + grp;
        a[i][0] = pack2(&As[r][ks + 2 * tig]);
        a[i][1] = pack2(&As[r + 8][ks + 2 * tig]);
        a[i][2] = pack2(&As[r][ks + 8 + 2 * tig]);
        a[i][3] = pack2(&As[r + 8][ks + 8 + 2 * tig]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = wn + 8 * j + grp;
        b[j][0] = pack2(&Bs[c][ks + 2 * tig]);
        b[j][1] = pack2(&Bs[c][ks + 8 + 2 * tig]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
              "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
              : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
              : "r"(a[i][0]), "r"(a[i][1]), "r"(a[i][2]), "r"(a[i][3]), "r"(b[j][0]), "r"(b[j][1]));
    }
    __syncthreads();
  }
  // epilogue: C fragment (row grp / grp + 8, columns 2 tig, 2 tig + 1)
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int m = m0 + wm + 16 * i + grp + (h >= 2 ? 8 : 0);
        const int n = n0 + wn + 8 * j + 2 * tig + (h & 1);
        if (m >= g.M || n >= g.N) continue;
        const long long o = (long long)m * g.ldc + n;
        float v = acc[i][j][h];
        if (g.bias) v += g.bias[n];
        if (g.act == 1) v = v > 0.f ? v : 0.f;
        if (g.act == 2 && !(__bfloat162float(g.mask[o]) > 0.f)) v = 0.f;
        if (g.act == 3) v = tanhf(v);
        if (g.act == 4) {
          const float a = __bfloat162float(g.mask[o]);
          v *= 1.f - a * a;
        }
        if (g.C32) g.C32[o] = g.beta != 0.f ? v + g.beta * g.C32[o] : v;
        if (g.C16) g.C16[o] = __float2bfloat16(v);
      }
}


// ---------------------------------------------------------------------------------------------
// pipelined path
constexpr int kPipeBN = 64, kPipeBK = 32, kStages = 3;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;  // 0: the 16 bytes are zero-filled, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

// Shared tile of one operand: R rows of W elements (+8 padding: rows 16 bytes out of bank step).
template <int R, int W>
struct STile {
  __nv_bfloat16 v[R][W + 8];
};

template <int TA, int TB, int BM>
struct PipeSmem {
  // A: [BM][BK] when K-contiguous (TA = 0), [BK][BM] when M-contiguous (TA = 1); B likewise.
  using ATile = STile<TA ? kPipeBK : BM, TA ? BM : kPipeBK>;
  using BTile = STile<TB ? kPipeBN : kPipeBK, TB ? kPipeBK : kPipeBN>;
  ATile a[kStages];
  BTile b[kStages];
};

template <int TA, int TB, int BM>
__device__ __forceinline__ void pipe_load(const GemmArgs& g, PipeSmem<TA, TB, BM>& sm, int slot, int k0, int m0,
                                          int n0) {
  const int tid = threadIdx.x;
  constexpr int kAChunks = BM * kPipeBK / 8, kBChunks = kPipeBN * kPipeBK / 8;
#pragma unroll
  for (int c = tid; c < kAChunks; c += 128) {
    int r, x, m, k;
    if (TA) {
      r = c / (BM / 8), x = (c % (BM / 8)) * 8, k = k0 + r, m = m0 + x;
    } else {
      r = c / (kPipeBK / 8), x = (c % (kPipeBK / 8)) * 8, m = m0 + r, k = k0 + x;
    }
    const bool ok = m < g.M && k < g.K;
    const __nv_bfloat16* src = ok ? (TA ? g.A + (long long)k * g.lda + m : g.A + (long long)m * g.lda + k) : g.A;
    cp_async16(smem_addr(&sm.a[slot].v[r][x]), src, ok);
  }
#pragma unroll
  for (int c = tid; c < kBChunks; c += 128) {
    int r, x, n, k;
    if (TB) {
      r = c / (kPipeBK / 8), x = (c % (kPipeBK / 8)) * 8, n = n0 + r, k = k0 + x;
    } else {
      r = c / (kPipeBN / 8), x = (c % (kPipeBN / 8)) * 8, k = k0 + r, n = n0 + x;
    }
    const bool ok = n < g.N && k < g.K;
    const __nv_bfloat16* src = ok ? (TB ? g.B + (long long)n * g.ldb + k : g.B + (long long)k * g.ldb + n) : g.B;
    cp_async16(smem_addr(&sm.b[slot].v[r][x]), src, ok);
  }
}

template <int TA, int TB, int BM>
__global__ void __launch_bounds__(128) gemm_pipe_kernel(const GemmArgs g0) {
  const GemmArgs g = at_group(g0);
  __shared__ __align__(128) PipeSmem<TA, TB, BM> sm;
  constexpr int MI = BM / 32;  // m16 tiles per warp (warp tile BM/2 x 32)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * kPipeBN;
  const int wm = (warp >> 1) * (BM / 2), wn = (warp & 1) * 32;
  float acc[MI][4][4] = {};
  const int nk = (g.K + kPipeBK - 1) / kPipeBK;
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nk) pipe_load<TA, TB, BM>(g, sm, s, s * kPipeBK, m0, n0);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2));
    __syncthreads();
    const int next = kt + kStages - 1;
    if (next < nk) pipe_load<TA, TB, BM>(g, sm, next % kStages, next * kPipeBK, m0, n0);
    asm volatile("cp.async.commit_group;\n" ::);
    const int slot = kt % kStages;
#pragma unroll
    for (int ks = 0; ks < kPipeBK; ks += 16) {
      uint32_t a[MI][4], b[4][2];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        if (TA) {
          const int k = ks + (lane & 7) + (lane >> 4) * 8, m = wm + 16 * i + ((lane >> 3) & 1) * 8;
          ldsm_x4_t(smem_addr(&sm.a[slot].v[k][m]), a[i]);
        } else {
          const int m = wm + 16 * i + (lane & 15), k = ks + (lane >> 4) * 8;
          ldsm_x4(smem_addr(&sm.a[slot].v[m][k]), a[i]);
        }
      }
#pragma unroll
      for (int jp = 0; jp < 2; ++jp) {
        uint32_t r[4];
        if (TB) {
          const int n = wn + 16 * jp + (lane & 7) + (lane >> 4) * 8, k = ks + ((lane >> 3) & 1) * 8;
          ldsm_x4(smem_addr(&sm.b[slot].v[n][k]), r);
        } else {
          const int k = ks + (lane & 7) + ((lane >> 3) & 1) * 8, n = wn + 16 * jp + (lane >> 4) * 8;
          ldsm_x4_t(smem_addr(&sm.b[slot].v[k][n]), r);
        }
        b[2 * jp][0] = r[0], b[2 * jp][1] = r[1], b[2 * jp + 1][0] = r[2], b[2 * jp + 1][1] = r[3];
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
              "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
              : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
              : "r"(a[i][0]), "r"(a[i][1]), "r"(a[i][2]), "r"(a[i][3]), "r"(b[j][0]), "r"(b[j][1]));
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  // epilogue: each thread holds column pairs (2 tig, 2 tig + 1) of rows grp and grp + 8
  const int grp = lane >> 2, tig = lane & 3;
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m0 + wm + 16 * i + grp + 8 * h;
        const int n = n0 + wn + 8 * j + 2 * tig;
        if (m >= g.M || n >= g.N) continue;  // N is a multiple of 8: n + 1 < N as well
        const long long o = (long long)m * g.ldc + n;
        float v0 = acc[i][j][2 * h], v1 = acc[i][j][2 * h + 1];
        if (g.bias) v0 += g.bias[n], v1 += g.bias[n + 1];
        if (g.act == 1) v0 = fmaxf(v0, 0.f), v1 = fmaxf(v1, 0.f);
        if (g.act == 2) {
          const __nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162*>(g.mask + o);
          if (!(__low2float(mk) > 0.f)) v0 = 0.f;
          if (!(__high2float(mk) > 0.f)) v1 = 0.f;
        }
        if (g.act == 3) v0 = tanhf(v0), v1 = tanhf(v1);
        if (g.act == 4) {
          const __nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162*>(g.mask + o);
          const float a0 = __low2float(mk), a1 = __high2float(mk);
          v0 *= 1.f - a0 * a0, v1 *= 1.f - a1 * a1;
        }
        if (g.C32) {
          float2* c = reinterpret_cast<float2*>(g.C32 + o);
          if (g.beta != 0.f) {
            const float2 old = *c;
            v0 += g.beta * old.x, v1 += g.beta * old.y;
          }
          *c = make_float2(v0, v1);
        }
        if (g.C16) *reinterpret_cast<__nv_bfloat162*>(g.C16 + o) = __floats2bfloat162_rn(v0, v1);
      }
}

template <int BM>
void launch_pipe(const GemmArgs& g, int groups, cudaStream_t s) {
  const dim3 grid((g.N + kPipeBN - 1) / kPipeBN, (g.M + BM - 1) / BM, groups);
  if (g.ta && g.tb) gemm_pipe_kernel<1, 1, BM><<<grid, 128, 0, s>>>(g);
  else if (g.ta) gemm_pipe_kernel<1, 0, BM><<<grid, 128, 0, s>>>(g);
  else if (g.tb) gemm_pipe_kernel<0, 1, BM><<<grid, 128, 0, s>>>(g);
  else gemm_pipe_kernel<0, 0, BM><<<grid, 128, 0, s>>>(g);
}

bool pipe_ok(const GemmArgs& g) {
  auto al = [](const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; };
  return g.M % 8 == 0 && g.N % 8 == 0 && g.K % 8 == 0 && g.lda % 8 == 0 && g.ldb % 8 == 0 && g.ldc % 2 == 0 &&
         g.sA % 8 == 0 && g.sB % 8 == 0 && g.sC % 2 == 0 && al(g.A, 16) && al(g.B, 16) && al(g.C32, 8) && al(g.C16, 4) && al(g.mask, 4);
}

// Column sums of an FP32 M x N matrix (bias gradients), per group (blockIdx.y: X and out move by
// xs and os elements). A block takes 32 columns; each of its 16 row lanes sums the rows lane,
// lane + 16, ... of one column (a warp reads 32 adjacent columns of one row), then lane 0 adds the
// 16 partial sums in lane order: a fixed order, so the result is the same on every run.
constexpr int kSumCols = 32, kSumLanes = 16;

__global__ void __launch_bounds__(kSumCols * kSumLanes) colsum_kernel(const float* X, int M, int N, int ld,
                                                                      long long xs, float* out, long long os) {
  __shared__ float part[kSumLanes][kSumCols + 1];
  X += blockIdx.y * xs;
  out += blockIdx.y * os;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int n = blockIdx.x * kSumCols + tx;
  float s = 0.f;
  if (n < N)
#pragma unroll 4
    for (int m = ty; m < M; m += kSumLanes) s += X[(long long)m * ld + n];
  part[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && n < N) {
    float t = 0.f;
    for (int q = 0; q < kSumLanes; ++q) t += part[q][tx];
    out[n] = t;
  }
}

// Mean-squared-error gradient of each group's mean over its M_g rows: G = (2 / (M_g N)) (Y - T),
// in FP32 and BF16; loss partials per row.
__global__ void mse_grad_kernel(const float* Y, const float* T, int Mg, int N, float* G32, __nv_bfloat16* G16,
                                float* row_loss) {
  const int m = blockIdx.x;
  float s = 0.f;
  const float scale = 2.f / ((float)Mg * (float)N);
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    const long long o = (long long)m * N + n;
    const float d = Y[o] - T[o];
    s += d * d;
    const float gr = scale * d;
    G32[o] = gr;
    G16[o] = __float2bfloat16(gr);
  }
  __shared__ float part[256];
  part[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int q = 0; q < (int)blockDim.x; ++q) t += part[q];
    row_loss[m] = t;
  }
}

// The same with the BF16 gradient transposed too (per group, N x M_g), in one pass: a block takes
// kMseRows rows of a group, a warp each, and walks the columns 128 at a time, the transposed part of
// kMseRows rows (16 bytes per column) going out through shared memory. 9 us for 2048 x 752 (24 MB, in
// L2; 6 steps in a row bound it); the two launches that this replaces took 17.
constexpr int kMseRows = 8, kMseCols = 128;

__global__ void __launch_bounds__(256) mse_grad_t_kernel(const float* Y, const float* T, int Mg, int N, float* G32,
                                                         __nv_bfloat16* G16, __nv_bfloat16* G16T, float* row_loss) {
  __shared__ __align__(16) __nv_bfloat16 tile[2][kMseCols][kMseRows];
  const int tid = threadIdx.x, ty = tid / 32, lane = tid % 32;
  const int r0 = blockIdx.x * kMseRows;  // Mg is a multiple of 8: every row is in
  const long long row = (long long)blockIdx.y * Mg + r0 + ty;
  const float scale = 2.f / ((float)Mg * (float)N);
  float s = 0.f;
  int half = 0;
  for (int c0 = 0; c0 < N; c0 += kMseCols, half ^= 1) {  // two tiles in turn: one barrier per step
    const int c = c0 + 4 * lane;
    if (c < N) {
      const long long o = row * N + c;
      const float4 y = *reinterpret_cast<const float4*>(Y + o), t = *reinterpret_cast<const float4*>(T + o);
      const float d[4] = {y.x - t.x, y.y - t.y, y.z - t.z, y.w - t.w};
      s += d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + d[3] * d[3];
      const float4 g = make_float4(scale * d[0], scale * d[1], scale * d[2], scale * d[3]);
      *reinterpret_cast<float4*>(G32 + o) = g;
      const __nv_bfloat162 lo = __floats2bfloat162_rn(g.x, g.y), hi = __floats2bfloat162_rn(g.z, g.w);
      *reinterpret_cast<uint2*>(G16 + o) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      __nv_bfloat16(*q)[kMseRows] = &tile[half][4 * lane];
      q[0][ty] = lo.x, q[1][ty] = lo.y, q[2][ty] = hi.x, q[3][ty] = hi.y;
    }
    __syncthreads();
    if (tid < kMseCols && c0 + tid < N)
      *reinterpret_cast<uint4*>(G16T + ((long long)blockIdx.y * N + c0 + tid) * Mg + r0) =
          *reinterpret_cast<const uint4*>(&tile[half][tid][0]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) row_loss[row] = s;
}

// Adam on FP32 master weights, with the BF16 copy the GEMMs read. The learning rate and the step
// number (for the bias corrections) are read from device memory, so that a captured training step
// replays unchanged while both move on.
__global__ void adam_kernel(float* w, __nv_bfloat16* w16, const float* grad, float* m1, float* m2, long long n,
                            const float* lr_dev, float b1, float b2, float eps, const int* step) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float t = (float)*step, lr = *lr_dev;
  const float c1 = 1.f - powf(b1, t), c2 = 1.f - powf(b2, t);
  const float g = grad[i];
  const float a = b1 * m1[i] + (1.f - b1) * g;
  const float b = b2 * m2[i] + (1.f - b2) * g * g;
  m1[i] = a;
  m2[i] = b;
  const float v = w[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
  w[i] = v;
  if (w16) w16[i] = __float2bfloat16(v);
}

__global__ void count_kernel(int* counter) { *counter += 1; }

// Adam on a whole network of every member, with its BF16 weights and their transposes: one launch in
// place of Adam, and a transpose per layer that read the BF16 weights back (8 members of 1.8 million
// parameters: 118 + 7 x 5 us before, of which two powf per parameter took Adam from its 66 us of
// memory traffic to 118). A block takes a 64 x 64 tile of one layer's weights (fan_in x fan_out): 16
// loads of 16 bytes per thread in flight, the updated tile through shared memory for the transpose.
// The blocks after a layer's tiles take its biases. blockIdx.y is the member. 80 us now, 7.0 TB/s. Run
// layer by layer beside the backward GEMMs it cost the step 20 us more than behind them: both want the
// same memory.
constexpr int kAdamLayers = 32, kAdamTile = 64;
struct AdamNet {
  int n;
  long long w[kAdamLayers], b[kAdamLayers];  // offsets of the weights and biases in a member's block
  int rows[kAdamLayers], cols[kAdamLayers];
  int first[kAdamLayers + 1];  // first block of each layer
};

struct AdamStep {
  float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ float adam_update(const AdamStep& t, float w, float g, float& m1, float& m2) {
  m1 = t.b1 * m1 + (1.f - t.b1) * g;
  m2 = t.b2 * m2 + (1.f - t.b2) * g * g;
  return w - t.lr * (m1 / t.c1) / (sqrtf(m2 / t.c2) + t.eps);
}

__global__ void __launch_bounds__(256) adam_net_kernel(const __grid_constant__ AdamNet net, float* w, __nv_bfloat16* w16,
                                                       __nv_bfloat16* w16t, const float* grad, float* m1, float* m2,
                                                       long long stride, const float* lr_dev, float b1, float b2,
                                                       float eps, const int* step) {
  __shared__ __align__(16) __nv_bfloat16 tile[kAdamTile][kAdamTile + 8];
  __shared__ AdamStep sh;
  const int tid = threadIdx.x;
  int l = 0;
  while (l + 1 < net.n && (int)blockIdx.x >= net.first[l + 1]) ++l;
  const int rows = net.rows[l], cols = net.cols[l];
  const int tc = (cols + kAdamTile - 1) / kAdamTile, tiles = tc * ((rows + kAdamTile - 1) / kAdamTile);
  const int blk = (int)blockIdx.x - net.first[l];
  const long long base = blockIdx.y * stride;
  // the step's constants (two powers: some microseconds of one thread) come behind the loads
  auto constants = [&] {
    if (tid == 0) {
      const float t = (float)*step;
      sh = AdamStep{*lr_dev, b1, b2, eps, 1.f - powf(b1, t), 1.f - powf(b2, t)};
    }
    __syncthreads();
    return sh;
  };
  if (blk >= tiles) {  // biases
    const AdamStep st = constants();
    const int i = (blk - tiles) * 256 + tid;
    if (i >= cols) return;
    const long long o = base + net.b[l] + i;
    float a = m1[o], b = m2[o];
    const float v = adam_update(st, w[o], grad[o], a, b);
    m1[o] = a, m2[o] = b, w[o] = v;
    w16[o] = __float2bfloat16(v);
    return;
  }
  const int r0 = blk / tc * kAdamTile, c0 = blk % tc * kAdamTile;
  const int tx = tid % 16, ty = tid / 16, c = c0 + 4 * tx;  // cols is a multiple of 8: a quad is in or out
  const long long o0 = base + net.w[l] + c;
  float4 g4[4], a4[4], b4[4], w4[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int r = r0 + ty + 16 * p;
    if (r >= rows || c >= cols) continue;
    const long long o = o0 + (long long)r * cols;
    g4[p] = *reinterpret_cast<const float4*>(grad + o);
    a4[p] = *reinterpret_cast<const float4*>(m1 + o);
    b4[p] = *reinterpret_cast<const float4*>(m2 + o);
    w4[p] = *reinterpret_cast<const float4*>(w + o);
  }
  const AdamStep st = constants();
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int r = r0 + ty + 16 * p;
    if (r >= rows || c >= cols) continue;
    const long long o = o0 + (long long)r * cols;
    w4[p].x = adam_update(st, w4[p].x, g4[p].x, a4[p].x, b4[p].x);
    w4[p].y = adam_update(st, w4[p].y, g4[p].y, a4[p].y, b4[p].y);
    w4[p].z = adam_update(st, w4[p].z, g4[p].z, a4[p].z, b4[p].z);
    w4[p].w = adam_update(st, w4[p].w, g4[p].w, a4[p].w, b4[p].w);
    *reinterpret_cast<float4*>(m1 + o) = a4[p];
    *reinterpret_cast<float4*>(m2 + o) = b4[p];
    *reinterpret_cast<float4*>(w + o) = w4[p];
    const __nv_bfloat162 lo = __floats2bfloat162_rn(w4[p].x, w4[p].y), hi = __floats2bfloat162_rn(w4[p].z, w4[p].w);
    *reinterpret_cast<uint2*>(w16 + o) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    const int row = ty + 16 * p;
    tile[4 * tx][row] = lo.x, tile[4 * tx + 1][row] = lo.y, tile[4 * tx + 2][row] = hi.x, tile[4 * tx + 3][row] = hi.y;
  }
  __syncthreads();
  // the transpose: column tid / 4 of the tile, 16 of its rows (rows is a multiple of 8)
  const int col = tid / 4, seg = tid % 4 * 16;
#pragma unroll
  for (int h = 0; h < 16; h += 8)
    if (c0 + col < cols && r0 + seg + h < rows)
      *reinterpret_cast<uint4*>(w16t + base + net.w[l] + (long long)(c0 + col) * rows + r0 + seg + h) =
          *reinterpret_cast<const uint4*>(&tile[col][seg + h]);
}

// One training batch in one launch, a block per (member, row): row idx[row] of the inputs as BF16, in
// rows and transposed (per member), and of the targets as FP32. Moves the step number on by one.
__global__ void __launch_bounds__(128) batch_kernel(const float* x, int n_in, const float* t, int n_out, const int* idx,
                                                    int rows, __nv_bfloat16* x16, __nv_bfloat16* x16t, float* t32,
                                                    int* counter) {
  const long long r = blockIdx.x;
  if (counter && r == 0 && threadIdx.x == 0) *counter += 1;
  const int member = (int)(r / rows), k = (int)(r - (long long)member * rows);
  const long long src = idx[r];
  for (int c = threadIdx.x; c < n_in; c += blockDim.x) {
    const __nv_bfloat16 v = __float2bfloat16(x[src * n_in + c]);
    x16[r * n_in + c] = v;
    x16t[((long long)member * n_in + c) * rows + k] = v;
  }
  const float4* s = reinterpret_cast<const float4*>(t + src * n_out);
  float4* d = reinterpret_cast<float4*>(t32 + r * n_out);
  for (int c = threadIdx.x; c < n_out / 4; c += blockDim.x) d[c] = s[c];
}

// An FP32 matrix of n elements as BF16, once per blockIdx.y.
__global__ void __launch_bounds__(256) replicate_kernel(const float* src, long long n, __nv_bfloat16* dst) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) dst[blockIdx.y * n + e] = __float2bfloat16(src[e]);
}

// The same from the launch's own parameters.
template <int N>
struct InlineInputs {
  float v[N];
};
template <int N>
__global__ void __launch_bounds__(256) replicate_inline_kernel(const __grid_constant__ InlineInputs<N> src, int n,
                                                               int copies, __nv_bfloat16* dst) {
  const int e = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (e >= n) return;
  const __nv_bfloat16 v = __float2bfloat16(src.v[e]);
  for (int k = 0; k < copies; ++k) dst[(long long)k * n + e] = v;
}

// Rows idx[0..rows) of an FP32 matrix with `cols` columns, into FP32 and/or BF16 copies.
__global__ void gather_kernel(const float* src, int cols, const int* idx, int rows, float* d32,
                              __nv_bfloat16* d16) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)rows * cols) return;
  const int r = (int)(e / cols), c = (int)(e % cols);
  const float v = src[(long long)idx[r] * cols + c];
  if (d32) d32[e] = v;
  if (d16) d16[e] = __float2bfloat16(v);
}

// dst (cols x rows, leading dimension ldd) = src^T (rows x cols, leading dimension lds), BF16,
// through 32 x 32 shared tiles (both sides coalesced); group blockIdx.z at ss / sd elements.
__global__ void transpose16_kernel(const __nv_bfloat16* src, int rows, int cols, int lds, long long ss,
                                   __nv_bfloat16* dst, int ldd, long long sd) {
  __shared__ __nv_bfloat16 t[32][33];
  src += blockIdx.z * ss;
  dst += blockIdx.z * sd;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    const int r = r0 + y, c = c0 + threadIdx.x;
    if (r < rows && c < cols) t[y][threadIdx.x] = src[(long long)r * lds + c];
  }
  __syncthreads();
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    const int c = c0 + y, r = r0 + threadIdx.x;
    if (r < rows && c < cols) dst[(long long)c * ldd + r] = t[threadIdx.x][y];
  }
}

// One GEMM launch of `groups` problems (blockIdx.z): the pipelined kernel where the shape and
// alignment allow, the scalar-staging kernel elsewhere. Returns 0 or -3 (launch error).
int gemm_grouped(const GemmArgs& g, int groups, cudaStream_t s, const char* who) {
  if (pipe_ok(g)) {
    // 64-row tiles unless that leaves fewer than two blocks per SM on a 152-SM part
    const long long tiles64 = (long long)((g.N + 63) / 64) * ((g.M + 63) / 64) * groups;
    if (tiles64 < 304) launch_pipe<32>(g, groups, s);
    else launch_pipe<64>(g, groups, s);
  } else {
    const dim3 grid((g.N + kBN - 1) / kBN, (g.M + kBM - 1) / kBM, groups);
    gemm_bf16_kernel<<<grid, 128, 0, s>>>(g);
  }
  const cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_last_error(std::string(who) + ": " + cudaGetErrorString(err));
    return -3;
  }
  return 0;
}

}  // namespace oafdtd

// --------------------------------------------------------------------------------------- C ABI
namespace {
// An asynchronous copy from a caller's memory that has been read when the scope ends, whatever the
// return path: mark() records an event on the stream, behind the copy and what was queued since, and the
// end waits for it. Not in a capture, which copies nothing yet.
struct CopyRead {
  cudaStream_t s = nullptr;
  cudaEvent_t ev = nullptr;
  bool pending = false;
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    s = stream;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaError_t err = cudaStreamIsCapturing(s, &cap);
    if (err == cudaSuccess) err = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
    pending = err == cudaSuccess && cap == cudaStreamCaptureStatusNone;
    return err;
  }
  void mark() {
    if (!pending || ev || cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return;
    if (cudaEventRecord(ev, s) != cudaSuccess) {
      cudaEventDestroy(ev);
      ev = nullptr;
    }
  }
  ~CopyRead() {
    if (!pending) return;
    if (ev) {
      cudaEventSynchronize(ev);
      cudaEventDestroy(ev);
    } else {
      cudaStreamSynchronize(s);
    }
  }
};

// n floats in host memory as BF16, `copies` times, read at the call.
template <int N>
cudaError_t replicate_inline(const float* x, int n, int copies, void* dst, cudaStream_t s) {
  oafdtd::InlineInputs<N> in;
  std::memcpy(in.v, x, (size_t)n * sizeof(float));
  oafdtd::replicate_inline_kernel<N>
      <<<(n + 255) / 256, 256, 0, s>>>(in, n, copies, static_cast<__nv_bfloat16*>(dst));
  return cudaGetLastError();
}
}  // namespace

extern "C" {

int oafdtd_mlp_transpose(const void* src, int32_t rows, int32_t cols, int32_t lds, void* dst, int32_t ldd,
                         int32_t groups, int64_t src_stride, int64_t dst_stride, void* stream) {
  if (!src || !dst || rows < 1 || cols < 1 || lds < cols || ldd < rows || groups < 1 || groups > 65535 ||
      (groups > 1 && (src_stride < (int64_t)rows * lds || dst_stride < (int64_t)cols * ldd))) {
    oafdtd::set_last_error("oafdtd_mlp_transpose: bad arguments");
    return -1;
  }
  const dim3 grid((cols + 31) / 32, (rows + 31) / 32, groups), block(32, 8);
  oafdtd::transpose16_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(src), rows, cols, lds, src_stride, static_cast<__nv_bfloat16*>(dst), ldd,
      dst_stride);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_gemm_tn(const void* A, const void* B, float* C32, void* C16, void* C16T, const float* bias,
                       const void* mask, int32_t M, int32_t N, int32_t K, int32_t lda, int32_t ldb, int32_t ldc,
                       int32_t ldct, int32_t act, float beta, int32_t groups, int64_t strideA, int64_t strideB,
                       int64_t strideC, int64_t strideCT, int64_t strideBias, int32_t* status, void* stream) {
  const bool bad_strides = groups > 1 && (strideA < (int64_t)M * lda || strideB < (int64_t)N * ldb ||
                                          ((C32 || C16 || mask) && strideC < (int64_t)M * ldc) ||
                                          (C16T && strideCT < (int64_t)N * ldct) || (bias && strideBias < N));
  if (!A || !B || (!C32 && !C16 && !C16T) || M < 1 || N < 1 || K < 1 || act < 0 || act > 4 ||
      ((act == 2 || act == 4) && !mask) || (C16T && ldct < M) || lda < K || ldb < K ||
      ((C32 || C16 || mask) && ldc < N) || groups < 1 || groups > 65535 || bad_strides) {
    oafdtd::set_last_error("oafdtd_mlp_gemm_tn: bad arguments");
    return -1;
  }
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  oafdtd::UmmaProblem p{A, B, C32, C16, C16T, bias, mask, M, N, K, lda, ldb, ldc, ldct, act, groups,
                        strideA, strideB, strideC, strideCT, strideBias, beta, status};
  // a transposed result whose rows TMA cannot address (ldct not a multiple of 8) is made from C16
  const bool own_t = C16T && C16 && !oafdtd::umma_shape_ok(p);
  if (own_t) p.C16T = nullptr;
  if (oafdtd::umma_shape_ok(p)) {
    std::string why;
    const cudaError_t err = oafdtd::launch_umma_gemm(p, s, &why);
    if (err == cudaSuccess)
      return own_t ? oafdtd_mlp_transpose(C16, M, N, ldc, C16T, ldct, groups, strideC, strideCT, stream) : 0;
    if (err != cudaErrorNotSupported) {
      oafdtd::set_last_error(std::string("oafdtd_mlp_gemm_tn: ") + (why.empty() ? cudaGetErrorString(err) : why));
      return -3;
    }
  }
  // other shapes: the mma.sync kernels (B transposed), then the transposed copy of the BF16 result
  if (C16T && !C16) {
    oafdtd::set_last_error("oafdtd_mlp_gemm_tn: a transposed result off the tcgen05 layouts needs C16 as well");
    return -1;
  }
  oafdtd::GemmArgs g;
  g.A = static_cast<const __nv_bfloat16*>(A);
  g.B = static_cast<const __nv_bfloat16*>(B);
  g.C32 = C32;
  g.C16 = static_cast<__nv_bfloat16*>(C16);
  g.bias = bias;
  g.mask = static_cast<const __nv_bfloat16*>(mask);
  g.M = M, g.N = N, g.K = K, g.lda = lda, g.ldb = ldb, g.ldc = ldc, g.ta = 0, g.tb = 1, g.act = act;
  g.beta = beta;
  g.sA = strideA, g.sB = strideB, g.sC = strideC, g.sBias = strideBias;
  int rc = oafdtd::gemm_grouped(g, groups, s, "oafdtd_mlp_gemm_tn");
  if (rc == 0 && C16T) rc = oafdtd_mlp_transpose(C16, M, N, ldc, C16T, ldct, groups, strideC, strideCT, stream);
  return rc;
}

int oafdtd_mlp_gemm(const void* A, const void* B, float* C32, void* C16, const float* bias, const void* mask,
                    int32_t M, int32_t N, int32_t K, int32_t lda, int32_t ldb, int32_t ldc, int32_t ta, int32_t tb,
                    int32_t act, float beta, void* stream) {
  if (!A || !B || (!C32 && !C16) || M < 1 || N < 1 || K < 1 || act < 0 || act > 4 || ((act == 2 || act == 4) && !mask)) {
    oafdtd::set_last_error("oafdtd_mlp_gemm: bad arguments");
    return -1;
  }
  oafdtd::GemmArgs g;
  g.A = static_cast<const __nv_bfloat16*>(A);
  g.B = static_cast<const __nv_bfloat16*>(B);
  g.C32 = C32;
  g.C16 = static_cast<__nv_bfloat16*>(C16);
  g.bias = bias;
  g.mask = static_cast<const __nv_bfloat16*>(mask);
  g.M = M, g.N = N, g.K = K, g.lda = lda, g.ldb = ldb, g.ldc = ldc, g.ta = ta, g.tb = tb, g.act = act;
  g.beta = beta;
  g.sA = g.sB = g.sC = g.sBias = 0;
  return oafdtd::gemm_grouped(g, 1, static_cast<cudaStream_t>(stream), "oafdtd_mlp_gemm");
}

int oafdtd_mlp_colsum(const float* X, int32_t M, int32_t N, int32_t ld, float* out, int32_t groups,
                      int64_t x_stride, int64_t out_stride, void* stream) {
  if (!X || !out || M < 1 || N < 1 || ld < N || groups < 1 || groups > 65535 ||
      (groups > 1 && (x_stride < (int64_t)M * ld || out_stride < N)))
    return -1;
  const dim3 block(oafdtd::kSumCols, oafdtd::kSumLanes), grid((N + oafdtd::kSumCols - 1) / oafdtd::kSumCols, groups);
  oafdtd::colsum_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(X, M, N, ld, x_stride, out,
                                                                                out_stride);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_mse_grad(const float* Y, const float* T, int32_t M, int32_t N, float* G32, void* G16,
                        float* row_loss, int32_t groups, void* stream) {
  if (!Y || !T || !G32 || !G16 || !row_loss || M < 1 || N < 1 || groups < 1 || M % groups != 0) return -1;
  oafdtd::mse_grad_kernel<<<M, 256, 0, static_cast<cudaStream_t>(stream)>>>(Y, T, M / groups, N, G32,
                                                                              static_cast<__nv_bfloat16*>(G16), row_loss);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_mse_grad_t(const float* Y, const float* T, int32_t M, int32_t N, float* G32, void* G16, void* G16T,
                          float* row_loss, int32_t groups, void* stream) {
  if (!Y || !T || !G32 || !G16 || !G16T || !row_loss || M < 1 || N < 1 || groups < 1 || groups > 65535 ||
      M % groups != 0)
    return -1;
  const int Mg = M / groups;
  bool fast = Mg % 8 == 0 && N % 8 == 0;
  for (const void* p : {static_cast<const void*>(Y), static_cast<const void*>(T), static_cast<const void*>(G32),
                        static_cast<const void*>(G16), static_cast<const void*>(G16T)})
    fast = fast && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
  if (!fast) {
    if (const int rc = oafdtd_mlp_mse_grad(Y, T, M, N, G32, G16, row_loss, groups, stream)) return rc;
    return oafdtd_mlp_transpose(G16, Mg, N, N, G16T, Mg, groups, (int64_t)Mg * N, (int64_t)Mg * N, stream);
  }
  oafdtd::mse_grad_t_kernel<<<dim3(Mg / oafdtd::kMseRows, groups), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      Y, T, Mg, N, G32, static_cast<__nv_bfloat16*>(G16), static_cast<__nv_bfloat16*>(G16T), row_loss);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_adam(float* w, void* w16, const float* grad, float* m1, float* m2, int64_t n, const float* lr,
                    float b1, float b2, float eps, const int32_t* step, void* stream) {
  if (!w || !grad || !m1 || !m2 || !lr || !step || n < 1) return -1;
  oafdtd::adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w, static_cast<__nv_bfloat16*>(w16), grad, m1, m2, n, lr, b1, b2, eps, step);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_adam_net(float* w, void* w16, void* w16t, const float* grad, float* m1, float* m2, int32_t n_layers,
                        const int64_t* layers, int32_t members, int64_t stride, const float* lr, float b1, float b2,
                        float eps, const int32_t* step, void* stream) {
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  bool ok = w && w16 && w16t && grad && m1 && m2 && layers && lr && step && n_layers >= 1 &&
            n_layers <= oafdtd::kAdamLayers && members >= 1 && members <= 65535 && stride % 8 == 0 && aligned(w) &&
            aligned(w16) && aligned(w16t) && aligned(grad) && aligned(m1) && aligned(m2);
  oafdtd::AdamNet net{};
  long long blocks = 0;
  for (int l = 0; ok && l < n_layers; ++l) {
    const int64_t* q = layers + 4 * l;  // weight offset, fan_in, fan_out, bias offset
    ok = q[0] >= 0 && q[0] % 8 == 0 && q[1] >= 1 && q[1] % 8 == 0 && q[2] >= 1 && q[2] % 8 == 0 && q[3] >= 0 &&
         q[0] + q[1] * q[2] <= stride && q[3] + q[2] <= stride && q[1] <= (1 << 20) && q[2] <= (1 << 20);
    net.w[l] = q[0], net.rows[l] = (int)q[1], net.cols[l] = (int)q[2], net.b[l] = q[3];
    net.first[l] = (int)blocks;
    blocks += ((q[1] + 63) / 64) * ((q[2] + 63) / 64) + (q[2] + 255) / 256;
    ok = ok && blocks <= 2147483647LL;
  }
  if (!ok) {
    oafdtd::set_last_error("oafdtd_mlp_adam_net: bad arguments");
    return -1;
  }
  net.n = n_layers;
  net.first[n_layers] = (int)blocks;
  oafdtd::adam_net_kernel<<<dim3((unsigned)blocks, members), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      net, w, static_cast<__nv_bfloat16*>(w16), static_cast<__nv_bfloat16*>(w16t), grad, m1, m2, stride, lr, b1, b2, eps,
      step);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_batch(const float* x, int32_t n_in, const float* t, int32_t n_out, const int32_t* idx, int32_t rows,
                     int32_t groups, void* x16, void* x16t, float* t32, int32_t* counter, void* stream) {
  if (!x || !t || !idx || !x16 || !x16t || !t32 || n_in < 1 || n_out < 4 || n_out % 4 != 0 || rows < 1 || groups < 1 ||
      (reinterpret_cast<uintptr_t>(t) & 15) || (reinterpret_cast<uintptr_t>(t32) & 15) ||
      (long long)rows * groups > 2147483647LL) {
    oafdtd::set_last_error("oafdtd_mlp_batch: bad arguments");
    return -1;
  }
  oafdtd::batch_kernel<<<(unsigned)(rows * groups), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      x, n_in, t, n_out, idx, rows, static_cast<__nv_bfloat16*>(x16), static_cast<__nv_bfloat16*>(x16t), t32, counter);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_gemm_list(const oafdtd_gemm* list, int32_t n, int32_t* status, void* stream) {
  if (!list || n < 1) {
    oafdtd::set_last_error("oafdtd_mlp_gemm_list: bad arguments");
    return -1;
  }
  for (int32_t at = 0; at < n;) {
    // as many as one launch takes, where every one suits it; else one by one
    oafdtd::UmmaProblem p[oafdtd::kUmmaList];
    int k = 0;
    for (; k < oafdtd::kUmmaList && at + k < n; ++k) {
      const oafdtd_gemm& q = list[at + k];
      p[k] = oafdtd::UmmaProblem{q.A, q.B, q.C32, nullptr, nullptr, nullptr, nullptr, q.M, q.N, q.K, q.lda, q.ldb,
                                 q.ldc, q.M, 0, q.groups, q.strideA, q.strideB, q.strideC, 0, 0, 0.f, status};
      if (!q.A || !q.B || !q.C32 || q.groups > 65535 || !oafdtd::umma_shape_ok(p[k])) break;
    }
    if (k > 1) {
      std::string why;
      const cudaError_t err = oafdtd::launch_umma_list(p, k, static_cast<cudaStream_t>(stream), &why);
      if (err == cudaSuccess) {
        at += k;
        continue;
      }
      if (err != cudaErrorNotSupported) {
        oafdtd::set_last_error(std::string("oafdtd_mlp_gemm_list: ") + (why.empty() ? cudaGetErrorString(err) : why));
        return -3;
      }
    }
    for (int end = at + (k > 1 ? k : 1); at < end; ++at) {
      const oafdtd_gemm& q = list[at];
      if (const int rc = oafdtd_mlp_gemm_tn(q.A, q.B, q.C32, nullptr, nullptr, nullptr, nullptr, q.M, q.N, q.K, q.lda,
                                            q.ldb, q.ldc, q.M, 0, 0.f, q.groups, q.strideA, q.strideB, q.strideC, 0, 0,
                                            status, stream))
        return rc;
    }
  }
  return 0;
}

static size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

// A prediction is a chain of one GEMM per layer, some 8 us each: 62 us for 412 rows of 8 members and seven
// layers. Layer by layer from Python, with the inputs' conversions and a buffer per layer from the
// framework, it took 200 us; from here, two activation buffers in turn, 125.
int64_t oafdtd_mlp_predict_bytes(int32_t rows, int32_t n_layers, const int64_t* layers, int32_t members) {
  if (rows < 1 || n_layers < 1 || !layers || members < 1) return 0;
  int64_t widest = 0;
  for (int l = 0; l + 1 < n_layers; ++l) widest = layers[4 * l + 2] > widest ? layers[4 * l + 2] : widest;
  const size_t n = (size_t)rows * (size_t)layers[1];
  return (int64_t)(align256(n * 4) + align256(n * 2 * members) + 2 * align256((size_t)rows * widest * 2 * members));
}

int oafdtd_mlp_predict(const float* x, int32_t rows, const float* p32, const void* w16t, int32_t n_layers,
                       const int64_t* layers, int32_t members, int64_t stride, int32_t act, void* work, float* y,
                       int64_t y_stride, int32_t* status, void* stream) {
  if (!x || rows < 1 || !p32 || !w16t || n_layers < 1 || !layers || members < 1 || members > 65535 || !work || !y) {
    oafdtd::set_last_error("oafdtd_mlp_predict: bad arguments");
    return -1;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t widest = 0;
  for (int l = 0; l + 1 < n_layers; ++l) widest = layers[4 * l + 2] > widest ? layers[4 * l + 2] : widest;
  const long long n = (long long)rows * layers[1];
  char* at = static_cast<char*>(work);
  float* x32 = reinterpret_cast<float*>(at);
  at += align256((size_t)n * 4);
  void* in = at;
  at += align256((size_t)n * 2 * members);
  void* act_buf[2] = {at, at + align256((size_t)rows * widest * 2 * members)};
  // The inputs have been read when the call returns: up to 16 KB as launch parameters (412 rows, eight
  // members: 119 us, as with a copy that nobody waits for; 122 with this wait), else by a copy that is
  // waited for (as launch parameters up to their limit of 32 KB: no faster, 161 us for 900 rows).
  CopyRead read;
  if (n <= 1024) {
    if (replicate_inline<1024>(x, (int)n, members, in, s) != cudaSuccess) return -3;
  } else if (n <= 4096) {
    if (replicate_inline<4096>(x, (int)n, members, in, s) != cudaSuccess) return -3;
  } else {
    if (read.copy(x32, x, (size_t)n * 4, s) != cudaSuccess) return -3;
    oafdtd::replicate_kernel<<<dim3((unsigned)((n + 255) / 256), members), 256, 0, s>>>(
        x32, n, static_cast<__nv_bfloat16*>(in));
    if (cudaGetLastError() != cudaSuccess) return -3;
  }
  for (int l = 0; l < n_layers; ++l) {
    const int64_t* q = layers + 4 * l;  // weight offset, fan_in, fan_out, bias offset
    const int a = (int)q[1], b = (int)q[2];
    const bool last = l == n_layers - 1;
    void* out = act_buf[l & 1];
    const int rc = oafdtd_mlp_gemm_tn(in, static_cast<const __nv_bfloat16*>(w16t) + q[0], last ? y : nullptr,
                                      last ? nullptr : out, nullptr, p32 + q[3], nullptr, rows, b, a, a, a, b, rows,
                                      last ? 0 : act, 0.f, members, (int64_t)rows * a, stride,
                                      last ? y_stride : (int64_t)rows * b, (int64_t)b * rows, stride, status, stream);
    if (rc != 0) return rc;
    if (l == n_layers / 2) read.mark();  // here the host is ahead of the device, and half the work is still to come
    in = out;
  }
  return 0;
}

int oafdtd_mlp_count(int32_t* counter, void* stream) {
  if (!counter) return -1;
  oafdtd::count_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(counter);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int oafdtd_mlp_gather(const float* src, int32_t cols, const int32_t* idx, int32_t rows, float* dst32, void* dst16,
                      void* stream) {
  if (!src || !idx || cols < 1 || rows < 1 || (!dst32 && !dst16)) return -1;
  const long long n = (long long)rows * cols;
  oafdtd::gather_kernel<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      src, cols, idx, rows, dst32, static_cast<__nv_bfloat16*>(dst16));
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // extern "C"
