// FDTD time-step kernels for sm_103a beside the sweeps (fused.cu, staged.cu, slab.cu).
//
//  * ghosts: PMC mirror planes, every wall in one launch.
//  * pre_e: H probe samples at (n + 1/2) dt; saves E^n of dispersive edges that also receive
//    injection (their ADE update runs after the injection, in the edge pass).
//  * sibc, edges: surface impedance on its edge list, then injection and the deferred Debye
//    updates on theirs.
//  * probe_e: E probe samples at (n + 1) dt.
//  * dft: the running DFTs of a chunk's samples, and the step counter.
// In variant 0 the direct sweeps take the samples and the injection with them (slab.cu).
//
// Arithmetic follows the reference engine (packages/oa-fdtd/src/oa_fdtd/reference.py:115-249)
// operation by operation; the library is built with -fmad=false, so float32 fields agree bit for
// bit with the float32 oracle. Fusing the CPML corrections into the sweeps keeps the reference's
// order (bulk update, then the corrections in ascending derivative axis, each rounded to the field
// precision), so fusion changes no rounding.

#include <algorithm>

#include "oafdtd_internal.cuh"
#include "probe.cuh"

namespace oafdtd {

// ----------------------------------------------------------------------------- PMC ghosts
// h[dst plane] = -h[src plane] for both components tangential to a PMC wall, over the whole plane
// (every storage index of the other axes), wall after wall in the order x low, x high, y low, ...
// One launch for every wall (blockIdx.y): where planes of two walls meet, the last wall's value
// follows from reflecting the point across each earlier wall it lies on, so no wall waits for
// another.
template <typename real>
struct GhostArgs {
  real* H[3];
  int mask, n[3], ext[3], B;
};

template <typename real>
__device__ __forceinline__ void ghost_wall(const GhostArgs<real>& g, int wall, int v, int u, int b) {
  const int axis = wall >> 1;
  const int u_ax = axis == 0 ? 1 : 0, v_ax = axis == 2 ? 1 : 2;
  const long long base = (long long)b * g.ext[0] * g.ext[1] * g.ext[2];
  for (int c = 0; c < 3; ++c) {
    if (c == axis) continue;
    int p[3];
    p[axis] = (wall & 1) ? g.n[axis] + 1 : 0;
    p[u_ax] = u;
    p[v_ax] = v;
    bool later = false;  // a later wall writes this point
    for (int w = wall + 1; w < 6; ++w)
      later |= ((g.mask >> w) & 1) && c != (w >> 1) && p[w >> 1] == ((w & 1) ? g.n[w >> 1] + 1 : 0);
    if (later) continue;
    const long long dst = base + ((long long)p[2] * g.ext[1] + p[1]) * g.ext[0] + p[0];
    bool neg = false;
    for (int w = wall; w >= 0; --w) {
      const int ax = w >> 1;
      if (!((g.mask >> w) & 1) || c == ax || p[ax] != ((w & 1) ? g.n[ax] + 1 : 0)) continue;
      p[ax] = (w & 1) ? g.n[ax] : 1;
      neg = !neg;
    }
    const real s = g.H[c][base + ((long long)p[2] * g.ext[1] + p[1]) * g.ext[0] + p[0]];
    g.H[c][dst] = neg ? -s : s;
  }
}

template <typename real>
__global__ void __launch_bounds__(256) ghost_kernel(const __grid_constant__ GhostArgs<real> g) {
  pdl_wait();
  const int wall = blockIdx.y, axis = wall >> 1;
  if (!((g.mask >> wall) & 1)) return;
  const int nu = g.ext[axis == 0 ? 1 : 0], nv = g.ext[axis == 2 ? 1 : 2];
  const long long total = (long long)nu * nv * g.B;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const long long r = t / nu;
    ghost_wall(g, wall, (int)(r % nv), (int)(t - r * nu), (int)(r / nv));
  }
}

// ----------------------------------------------------------------------------- probes
// Every step's probe samples (probe_sample) are kept for the chunk; one launch at its end adds
// them to the running DFTs, acc[f] += exp(-j w t) dt V with t = (n + offset) dt, step after step as
// the reference does, and advances the step counter. In variant 0 the sweeps take every sample but the last
// step's E probes, which this launch takes. A DFT per step put 256 float64 sincos of one
// block on the path of every step (8 us a step for the E probes at 64 to 256 frequencies: GB300
// issues two float64 operations a clock and SM); here a block takes four frequencies, one thread
// per (frequency, step) for the phases, which all probes of a kind share, then one thread per
// (probe, member, frequency) for the sums.
constexpr int kDftF = 4;

// Blocks of a DFT launch; tail: it takes the last step's E samples first, a block each.
template <typename real>
__host__ __device__ __forceinline__ int dft_blocks_of(const ProbeArgs<real>& a, bool tail) {
  return (a.n_probe > 0 && a.n_freq > 0 ? 2 * ((a.n_freq + kDftF - 1) / kDftF) : 1) + (tail ? a.n_kind[0] * a.B : 0);
}

// Steps base .. base + n - 1 of the probes of the kinds in `kinds` (bit 0 E, bit 1 H). tail: the last
// step's E samples are not in yet. The first blocks take one each, the others leave them out of their
// sums, and the block that ends last adds them. (Every block taking them all, one after the other: a single
// step with 30 probes of 11932 points 4150 us at 200x160x80, 209 now, 156 with port probes alone.)
template <typename real>
__device__ __forceinline__ void dft_body(const ProbeArgs<real>& a, int block, int n, int kinds, bool tail, int bump) {
  __shared__ double2 ph[kDftF][kChunk];
  __shared__ int last;
  const long long base = *a.step_base;
  const int tails = tail ? a.n_kind[0] * a.B : 0, tid = (int)threadIdx.x;
  if (block < tails) {
    probe_sample(a, 0, block, n - 1);
  } else {
    const int nfb = (a.n_freq + kDftF - 1) / kDftF, d = block - tails;
    const int kind = nfb > 0 ? d / nfb : 0, f0 = nfb > 0 ? (d % nfb) * kDftF : 0;
    const int pairs = (kinds >> kind) & 1 ? a.n_kind[kind] * a.B : 0;
    if (pairs > 0 && a.n_freq > 0) {
      const int fi = tid / kChunk, o = tid % kChunk, m = tail && kind == 0 ? n - 1 : n;
      if (o < n && f0 + fi < a.n_freq) {
        const double t = ((double)(base + o) + (kind == 0 ? 1.0 : 0.5)) * a.dt;
        double sn, cs;
        sincos(a.omega[f0 + fi] * t, &sn, &cs);
        ph[fi][o] = make_double2(cs * a.dt, -(sn * a.dt));
        if (o >= m) a.tail_phase[f0 + fi] = ph[fi][o];
      }
      __syncthreads();
      const int f = tid % kDftF;
      for (int q = tid / kDftF; q < pairs && f0 + f < a.n_freq && m > 0; q += kChunk) {
        const long long pb = (long long)a.list[kind][q / a.B] * a.B + q % a.B;
        const double* v = a.vals + pb * kChunk;
        double2* out = a.acc + pb * a.n_freq + f0 + f;
        double2 cur = *out;
#pragma unroll 8
        for (int s = 0; s < m; ++s) {
          const double x = v[s];
          cur.x += ph[f][s].x * x;
          cur.y += ph[f][s].y * x;
        }
        *out = cur;
      }
    }
  }
  if (bump == 0) return;
  // the last block to get here advances the counter: every block has read it, and its work is done
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    last = atomicAdd(a.dft_done, 1) == dft_blocks_of(a, tail) - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int terms = tails * a.n_freq;  // the accumulators of one kind: below 2^31 elements in memory
  constexpr int kAhead = 8, kStep = kDftF * kChunk;
  for (int e0 = tid; e0 < terms; e0 += kAhead * kStep) {
    double2* out[kAhead];
    double2 cur[kAhead], p[kAhead];
    double x[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int e = min(e0 + u * kStep, terms - 1), q = e / a.n_freq, f = e - q * a.n_freq;
      const long long pb = (long long)a.list[0][q / a.B] * a.B + q % a.B;
      x[u] = __ldcg(a.vals + pb * kChunk + n - 1);
      p[u] = __ldcg(a.tail_phase + f);
      out[u] = a.acc + pb * a.n_freq + f;
      cur[u] = __ldcg(out[u]);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (e0 + u * kStep >= terms) continue;
      cur[u].x += p[u].x * x[u];
      cur[u].y += p[u].y * x[u];
      *out[u] = cur[u];
    }
  }
  if (tid == 0) {
    *a.dft_done = 0;
    *a.counter += bump;
  }
}

template <typename real>
__global__ void __launch_bounds__(kDftF* kChunk) dft_kernel(const __grid_constant__ ProbeArgs<real> a, int n, int kinds,
                                                            int tail, int bump) {
  pdl_wait();
  dft_body(a, (int)blockIdx.x, n, kinds, tail != 0, bump);
}

// Several engines' DFTs (and step counters) in one launch.
template <typename real>
__global__ void __launch_bounds__(kDftF* kChunk)
    dft_batch_kernel(const ProbeArgs<real>* __restrict__ A, const BatchGrid G, int n, int tail) {
  __shared__ __align__(16) unsigned char args[sizeof(ProbeArgs<real>)];
  int e;
  const uint3 bid = G.block(&e);
  const ProbeArgs<real>& a = stage_args(A + e, args);
  pdl_wait();
  dft_body(a, (int)bid.x, n, 3, tail != 0, n);
}

template <typename real>
__device__ __forceinline__ void pre_e_body(const ProbeArgs<real>& a, int off, int block) {
  const int nprobe_blocks = a.n_kind[1] * a.B;
  if (block < nprobe_blocks) {
    probe_sample(a, 1, block, off);
    return;
  }
  const int t = (block - nprobe_blocks) * blockDim.x + threadIdx.x;
  if (t >= a.n_def) return;
  const real* E = a.E[a.def_comp[t]];
  for (int b = 0; b < a.B; ++b) a.eold[(long long)b * a.n_def + t] = E[(long long)b * a.bs + a.def_flat[t]];
}

template <typename real>
__global__ void __launch_bounds__(256) pre_e_kernel(const __grid_constant__ ProbeArgs<real> a, int off) {
  pre_e_body(a, off, (int)blockIdx.x);
}

template <typename real>
__global__ void __launch_bounds__(256) probe_e_kernel(const __grid_constant__ ProbeArgs<real> a, int off) {
  probe_sample(a, 0, (int)blockIdx.x, off);
}

// Several engines' deferred-E saves and H-probe samples, and E-probe samples, in one launch each.
template <typename real>
__global__ void __launch_bounds__(256) pre_e_batch_kernel(const ProbeArgs<real>* __restrict__ A, const BatchGrid G,
                                                          int off) {
  __shared__ __align__(16) unsigned char args[sizeof(ProbeArgs<real>)];
  int e;
  const uint3 bid = G.block(&e);
  pre_e_body(stage_args(A + e, args), off, (int)bid.x);
}

template <typename real>
__global__ void __launch_bounds__(256) probe_e_batch_kernel(const ProbeArgs<real>* __restrict__ A, const BatchGrid G,
                                                            int off) {
  __shared__ __align__(16) unsigned char args[sizeof(ProbeArgs<real>)];
  int e;
  const uint3 bid = G.block(&e);
  probe_sample(stage_args(A + e, args), 0, (int)bid.x, off);
}

// ----------------------------------------------------------------------------- surface impedance
// E_face = r0 J + sum_p v_p, v_p = alpha_p (J - J_prev) + g_p v_p, J = sum of the signed outside
// H samples (reference.py:129-150). A thread handles the batch members of an edge (kSibcMembers); BB and PP
// unroll the batch and pole loops so all loads of an edge are issued together.
// Members of one edge that a thread takes, of BB in all: all of them in float32 (one per thread 146 us
// against 123 for 1.9 million edges, two members); one in float64, where two take 190 registers and
// four 254 with spills (84 against 92 us for 0.27 million edges, two members).
template <typename real, int BB>
constexpr int kSibcMembers = sizeof(real) == 4 ? BB : (BB < 1 ? BB : 1);

template <typename real, int BB, int PP>
__device__ __forceinline__ void sibc_body(const SibcArgs<real>& a, int block, int lo, int hi) {
  constexpr int N = kSibcMembers<real, BB>;
  int b0 = 0;
  if constexpr (N < BB) {  // the members of an edge in blocks side by side
    b0 = block % BB;
    block /= BB;
  }
  const int s = lo + block * (int)blockDim.x + (int)threadIdx.x;
  if (s >= hi) return;
  const SibcEdge<real> ed = a.edge[s];
  const real* __restrict__ alpha = a.alpha + (long long)ed.mat * PP;
  const long long n = a.n;
  // every load of this edge first (the stores below would otherwise order them one by one)
  real vv[N][PP], hs[N][2], jp[N];
#pragma unroll
  for (int b = 0; b < N; ++b) {
    const long long off = (long long)(b0 + b) * a.bs;
    const long long be = (long long)(b0 + b) * n + s;
    hs[b][0] = ed.sign[0] != (real)0 ? a.H[ed.hcomp0][off + ed.hflat[0]] : (real)0;
    hs[b][1] = ed.sign[1] != (real)0 ? a.H[ed.hcomp1][off + ed.hflat[1]] : (real)0;
    jp[b] = a.jprev[be];
#pragma unroll
    for (int p = 0; p < PP; ++p) vv[b][p] = a.v[((long long)p * BB) * n + be];
  }
  const real r0 = a.r0[ed.mat];
#pragma unroll
  for (int b = 0; b < N; ++b) {
    real jj = (real)0;
    if (ed.sign[0] != (real)0) jj = jj + ed.sign[0] * hs[b][0];
    if (ed.sign[1] != (real)0) jj = jj + ed.sign[1] * hs[b][1];
    const real dj = jj - jp[b];
    real vsum = (real)0;
#pragma unroll
    for (int p = 0; p < PP; ++p) {
      const real nv = alpha[p] * dj + a.gp[p] * vv[b][p];
      vv[b][p] = nv;
      vsum = p == 0 ? nv : vsum + nv;
    }
    const long long be = (long long)(b0 + b) * n + s;
#pragma unroll
    for (int p = 0; p < PP; ++p) a.v[((long long)p * BB) * n + be] = vv[b][p];
    a.jprev[be] = jj;
    a.E[ed.comp][(long long)(b0 + b) * a.bs + ed.flat] = r0 * jj + vsum;
  }
}

template <typename real, int BB, int PP>
__global__ void __launch_bounds__(128) sibc_kernel(const __grid_constant__ SibcArgs<real> a, int lo, int hi) {
  pdl_wait();
  sibc_body<real, BB, PP>(a, (int)blockIdx.x, lo, hi);
}

// Any batch size and pole count (loops not unrolled).
template <typename real>
__device__ __forceinline__ void sibc_generic_body(const SibcArgs<real>& a, int block, int lo, int hi) {
  const int s = lo + block * (int)blockDim.x + (int)threadIdx.x;
  if (s >= hi) return;
  const SibcEdge<real> ed = a.edge[s];
  const int B = a.B, P = a.P;
  const real* __restrict__ alpha = a.alpha + (long long)ed.mat * P;
  const long long n = a.n;
  for (int b = 0; b < B; ++b) {
    const long long off = (long long)b * a.bs;
    real jj = (real)0;
    if (ed.sign[0] != (real)0) jj = jj + ed.sign[0] * a.H[ed.hcomp0][off + ed.hflat[0]];
    if (ed.sign[1] != (real)0) jj = jj + ed.sign[1] * a.H[ed.hcomp1][off + ed.hflat[1]];
    const long long be = (long long)b * n + s;
    const real dj = jj - a.jprev[be];
    real vsum = (real)0;
    for (int p = 0; p < P; ++p) {
      real* vp = a.v + ((long long)p * B) * n + be;
      const real nv = alpha[p] * dj + a.gp[p] * (*vp);
      *vp = nv;
      vsum = p == 0 ? nv : vsum + nv;
    }
    a.jprev[be] = jj;
    a.E[ed.comp][off + ed.flat] = a.r0[ed.mat] * jj + vsum;
  }
}

template <typename real>
__global__ void __launch_bounds__(128) sibc_generic_kernel(const __grid_constant__ SibcArgs<real> a, int lo, int hi) {
  pdl_wait();
  sibc_generic_body(a, (int)blockIdx.x, lo, hi);
}

// Several engines' surface-impedance updates in one launch (engines of one kernel variant).
template <typename real, int BB, int PP>
__global__ void __launch_bounds__(128) sibc_batch_kernel(const SibcArgs<real>* __restrict__ A, const BatchGrid G) {
  __shared__ __align__(16) unsigned char args[sizeof(SibcArgs<real>)];
  int e;
  const uint3 bid = G.block(&e);
  const SibcArgs<real>& a = stage_args(A + e, args);
  pdl_wait();
  if constexpr (BB == 0)
    sibc_generic_body(a, (int)bid.x, 0, a.n);
  else
    sibc_body<real, BB, PP>(a, (int)bid.x, 0, a.n);
}

template <typename real>
int sibc_variant(const SibcArgs<real>& a) {
  return a.P == 16 && (a.B == 1 || a.B == 2 || a.B == 4) ? a.B : 0;
}

// Blocks of 128 threads for n edges.
template <typename real>
int sibc_blocks_of(const SibcArgs<real>& a, int n) {
  const int split = sizeof(real) == 8 ? std::max(sibc_variant(a), 1) : 1;  // BB / kSibcMembers
  return (n + 127) / 128 * split;
}

template <typename real>
int sibc_blocks(const SibcArgs<real>& a) {
  return sibc_blocks_of(a, a.n);
}

template <typename real>
cudaError_t launch_sibc_batch(const SibcArgs<real>* A, const BatchGrid& G, int blocks, int variant, bool pdl,
                              cudaStream_t s) {
  if (blocks <= 0) return cudaSuccess;
  auto kernel = variant == 2   ? sibc_batch_kernel<real, 2, 16>
                : variant == 1 ? sibc_batch_kernel<real, 1, 16>
                : variant == 4 ? sibc_batch_kernel<real, 4, 16>
                               : sibc_batch_kernel<real, 0, 16>;
  return launch_pdl(pdl, kernel, dim3(blocks), dim3(128), 0, s, A, G);
}

template <typename real>
cudaError_t launch_sibc(const SibcArgs<real>& a, cudaStream_t s, int lo, int hi, bool pdl) {
  if (hi < 0) hi = a.n;
  if (hi <= lo) return cudaSuccess;
  const int variant = sibc_variant(a);
  auto kernel = variant == 2   ? sibc_kernel<real, 2, 16>
                : variant == 1 ? sibc_kernel<real, 1, 16>
                : variant == 4 ? sibc_kernel<real, 4, 16>
                               : sibc_generic_kernel<real>;
  return launch_pdl(pdl, kernel, dim3((unsigned)sibc_blocks_of(a, hi - lo)), dim3(128), 0, s, a, lo, hi);
}

// ----------------------------------------------------------------------------- injection pass
// Injection (reference.py:223-234) and the Debye update of dispersive edges with injection
// (reference.py:119-127), in the reference's order after the surface impedance.
template <typename real>
__device__ __forceinline__ void edge_body(const EdgeArgs<real>& a, int off, int block) {
  const int e = block * blockDim.x + threadIdx.x;
  if (e >= a.n) return;
  const long long step = *a.step_base + off;
  const int c = a.comp[e];
  const long long f = a.flat[e];
  const int ib = a.inj_beg[e], ie = a.inj_end[e];
  const int ds = a.def_slot[e];
  for (int b = 0; b < a.B; ++b) {
    real* Ec = a.E[c] + (long long)b * a.bs;
    real val = Ec[f];
    for (int t = ib; t < ie; ++t) {
      const int ch = a.i_chan[t];
      const double w = a.wave[(long long)ch * a.max_steps + step];
      val = val + (real)((a.drive[b * a.n_chan + ch] * w) * a.i_amp[t]);
    }
    if (ds >= 0) {
      const long long q = f;
      const int m = a.mat[c][q];
      const int kk = (int)(q / ((long long)a.X * a.Y));
      const long long rem = q - (long long)kk * a.X * a.Y;
      const long long jstride = (long long)a.B * a.jnk[c] * a.Y * a.X;
      const long long jq = ((long long)b * a.jnk[c] + (kk - a.jk0[c])) * a.Y * a.X + rem;
      real* J = a.J[c];
      const int AP = a.ade_P;
      real jt = (real)0;
      for (int p = 0; p < AP; ++p) jt = jt + a.ade_onekp[p] * J[jq + p * jstride];
      jt = (real)0.5 * jt;
      const real en = val - a.coef[m].cbe * jt;
      const real de = en - a.eold[(long long)b * a.n_def + ds];
      for (int p = 0; p < AP; ++p) {
        const long long qq = jq + p * jstride;
        const real beta = p == 0 ? a.coef[m].beta0 : a.ade_beta[(long long)m * AP + p];
        J[qq] = a.ade_kp[p] * J[qq] + beta * de;
      }
      val = en;
    }
    Ec[f] = val;
  }
}

template <typename real>
__global__ void __launch_bounds__(128) edge_kernel(const __grid_constant__ EdgeArgs<real> a, int off) {
  edge_body(a, off, (int)blockIdx.x);
}

// Several engines' injection passes in one launch.
template <typename real>
__global__ void __launch_bounds__(128) edge_batch_kernel(const EdgeArgs<real>* __restrict__ A, const BatchGrid G,
                                                         int off) {
  __shared__ __align__(16) unsigned char args[sizeof(EdgeArgs<real>)];
  int e;
  const uint3 bid = G.block(&e);
  edge_body(stage_args(A + e, args), off, (int)bid.x);
}

// ----------------------------------------------------------------------------- energy
// Float-float arithmetic (a value is hi + lo, two float32 with |lo| <= ulp(hi) / 2): products
// from the float32 multiply and its exact error (one fused multiply-add, written out: the
// library is built without contraction), sums by Knuth's two-sum. About 2^-46 relative error
// per operation.
__device__ __forceinline__ float2 ff_mul(float2 a, float2 b) {
  const float p = a.x * b.x;
  float e = __fmaf_rn(a.x, b.x, -p);
  e = __fmaf_rn(a.x, b.y, e);
  e = __fmaf_rn(a.y, b.x, e);
  const float s = p + e;
  return make_float2(s, e - (s - p));
}
__device__ __forceinline__ float2 ff_add(float2 a, float2 b) {
  const float s = a.x + b.x;
  const float bb = s - a.x;
  const float err = (a.x - (s - bb)) + (b.x - bb);
  const float lo = (err + a.y) + b.y;
  const float h = s + lo;
  return make_float2(h, lo - (h - s));
}

// The sum of v^2 w over four cells, as a float-float pair. Products are exact to 2^-46, their rounded
// parts are summed with the errors gathered apart (four of them: the gathered part needs no carry).
__device__ __forceinline__ float2 ff_quad(const float v[4], const float2 w[4]) {
  float hi = 0.0f, lo = 0.0f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float p = v[e] * v[e];
    const float h = w[e].x * p;
    lo = __fmaf_rn(w[e].y, p, __fmaf_rn(w[e].x, __fmaf_rn(v[e], v[e], -p), lo)) + __fmaf_rn(w[e].x, p, -h);
    const float s = hi + h, bb = s - hi;
    lo += (hi - (s - bb)) + (h - bb);
    hi = s;
  }
  const float s = hi + lo;
  return make_float2(s, lo - (s - hi));
}

// Energy sums 1/2 sum eps E^2 V (and sum H^2 V) per component, in float64 or, for float32
// fields, in float-float: GB300's float64 rate is a small fraction of its float32 rate, and a
// float64 product chain per cell makes this kernel compute-bound (3.3 ms at 400x400x120, batch
// 2; the fields are read in 0.15 ms). A float32 field value squares exactly into a float-float
// pair; the weights come as float-float pairs; the terms of a thread are summed in float-float
// and the thread's sum converted to float64 once. Each term is then exact to about 1e-13 relative,
// so the sum is too (every term is positive). The fields are scaled by 2^32 and the weights by
// 2^40 (exact) so that squares of fields down to 1e-28 and weights down to 1e-30 stay normal;
// the thread's sum is scaled back by 2^-104. Fields above 4e9 would overflow the square.
// Field and weights of 38 million cells (1.1 GB, 0.16 ms) take 0.45 ms, 0.61 before: bound by the
// instructions of the pairs (about 130 per quad).
// A thread takes a quad (four cells of a row) per turn. The y-z weight, and the permittivity where
// the four cells have one, multiply the quad's sum instead of each cell: a third of the float-float
// operations. The quads of a thread lie a grid apart, and row and column move on by adding.
template <typename real>
__global__ void __launch_bounds__(256, 4) energy_kernel(const __grid_constant__ EnergyArgs<real> a,
                                                        double* partial) {
  __shared__ double warp_sum[8];
  const int cc = blockIdx.y;  // 0..2 E, 3..5 H
  const real* F = a.F[cc];
  const ushort4* M = cc < 3 ? reinterpret_cast<const ushort4*>(a.mat[cc]) : nullptr;
  const int Q = a.X / 4;
  const long long rows = (long long)a.Z * a.Y, per = rows * Q, quads = per * a.B;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long dr = stride / Q;
  const int dq = (int)(stride - dr * Q);
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long r = t / Q;  // row of the member
  int i = (int)(t - r * Q);
  long long base = 0;  // first quad of the member
  double acc = 0.0;
  auto settle = [&] {  // r into its member
    while (r >= rows) r -= rows, base += per;
  };
  auto advance = [&] {
    t += stride, r += dr, i += dq;
    if (i >= Q) i -= Q, ++r;
    settle();
  };
  settle();
  if constexpr (sizeof(real) == 4) {
    const float vscale = ldexpf(1.0f, kEnergyVShift);
    const float4* wx4 = reinterpret_cast<const float4*>(a.wxf[cc]);
    const float2* wyzf = a.wyzf[cc];
    float2 sum = make_float2(0.0f, 0.0f);
    for (; t < quads; advance()) {
      const float4 f = reinterpret_cast<const float4*>(F)[t], w01 = wx4[2 * i], w23 = wx4[2 * i + 1];
      const float2 wyz = wyzf[r];
      const float v[4] = {f.x * vscale, f.y * vscale, f.z * vscale, f.w * vscale};
      float2 w[4] = {{w01.x, w01.y}, {w01.z, w01.w}, {w23.x, w23.y}, {w23.z, w23.w}};
      float2 q;
      if (M) {
        const ushort4 m = M[t - base];
        if (m.x == m.y && m.x == m.z && m.x == m.w) {
          q = ff_mul(ff_quad(v, w), a.epsf[m.x]);
        } else {
          w[0] = ff_mul(w[0], a.epsf[m.x]), w[1] = ff_mul(w[1], a.epsf[m.y]);
          w[2] = ff_mul(w[2], a.epsf[m.z]), w[3] = ff_mul(w[3], a.epsf[m.w]);
          q = ff_quad(v, w);
        }
      } else {
        q = ff_quad(v, w);
      }
      sum = ff_add(sum, ff_mul(q, wyz));
    }
    acc = ldexp((double)sum.x + (double)sum.y, -(kEnergyVShift * 2 + kEnergyWShift));
  } else {
    const double* wx = a.w[cc][0];
    const double* wy = a.w[cc][1];
    const double* wz = a.w[cc][2];
    for (; t < quads; advance()) {
      const double2 f = reinterpret_cast<const double2*>(F)[2 * t], g = reinterpret_cast<const double2*>(F)[2 * t + 1];
      const int k = (int)(r / a.Y), j = (int)(r - (long long)k * a.Y);
      double w[4] = {wx[4 * i], wx[4 * i + 1], wx[4 * i + 2], wx[4 * i + 3]};
      if (M) {
        const ushort4 m = M[t - base];
        w[0] *= a.eps[m.x], w[1] *= a.eps[m.y], w[2] *= a.eps[m.z], w[3] *= a.eps[m.w];
      }
      const double q = w[0] * (f.x * f.x) + w[1] * (f.y * f.y) + (w[2] * (g.x * g.x) + w[3] * (g.y * g.y));
      acc += wy[j] * wz[k] * q;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += warp_sum[w];
    partial[(long long)cc * gridDim.x + blockIdx.x] = s;
  }
}

// A warp per component, in a fixed order (one thread per component took 130 us over 1216 partials,
// each addition behind its load).
__global__ void __launch_bounds__(192) energy_final_kernel(const double* partial, int nblocks, double* out) {
  const int cc = threadIdx.x / 32, lane = threadIdx.x % 32;
  double s = 0.0;
#pragma unroll 4
  for (int k = lane; k < nblocks; k += 32) s += partial[(long long)cc * nblocks + k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[cc] = s;
}

// ----------------------------------------------------------------------------- launchers
static inline unsigned ceil_div(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

template <typename real>
cudaError_t launch_ghosts(real* const H[3], int pmc_mask, int nx, int ny, int nz, int X, int Y, int B,
                          cudaStream_t s, bool pdl) {
  GhostArgs<real> g{{H[0], H[1], H[2]}, pmc_mask, {nx, ny, nz}, {X, Y, nz + 2}, B};
  long long most = 0;
  for (int w = 0; w < 6; ++w)
    if ((pmc_mask >> w) & 1) {
      const int axis = w >> 1;
      most = std::max(most, (long long)g.ext[axis == 0 ? 1 : 0] * g.ext[axis == 2 ? 1 : 2] * B);
    }
  if (most == 0) return cudaSuccess;
  return launch_pdl(pdl, ghost_kernel<real>, dim3(std::min(ceil_div(most, 256), 152u * 8u), 6), dim3(256), 0, s, g);
}

template <typename real>
int pre_e_blocks(const ProbeArgs<real>& a) {
  return a.n_kind[1] * a.B + (int)ceil_div(a.n_def, 256);
}

template <typename real>
int probe_e_blocks(const ProbeArgs<real>& a) {
  return a.n_kind[0] * a.B;
}

template <typename real>
int edge_blocks(const EdgeArgs<real>& a) {
  return a.n == 0 ? 0 : (int)ceil_div(a.n, 128);
}

template <typename real>
cudaError_t launch_pre_e_batch(const ProbeArgs<real>* A, const BatchGrid& G, int blocks, int off, cudaStream_t s) {
  if (blocks <= 0) return cudaSuccess;
  pre_e_batch_kernel<real><<<blocks, 256, 0, s>>>(A, G, off);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_probe_e_batch(const ProbeArgs<real>* A, const BatchGrid& G, int blocks, int off, cudaStream_t s) {
  if (blocks <= 0) return cudaSuccess;
  probe_e_batch_kernel<real><<<blocks, 256, 0, s>>>(A, G, off);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_edges_batch(const EdgeArgs<real>* A, const BatchGrid& G, int blocks, int off, cudaStream_t s) {
  if (blocks <= 0) return cudaSuccess;
  edge_batch_kernel<real><<<blocks, 128, 0, s>>>(A, G, off);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_pre_e(const ProbeArgs<real>& a, int off, cudaStream_t s) {
  const int blocks = pre_e_blocks(a);
  if (blocks == 0) return cudaSuccess;
  pre_e_kernel<real><<<blocks, 256, 0, s>>>(a, off);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_probe_e(const ProbeArgs<real>& a, int off, cudaStream_t s) {
  const int blocks = a.n_kind[0] * a.B;
  if (blocks == 0) return cudaSuccess;
  probe_e_kernel<real><<<blocks, 256, 0, s>>>(a, off);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_edges(const EdgeArgs<real>& a, int off, cudaStream_t s) {
  if (a.n == 0) return cudaSuccess;
  edge_kernel<real><<<ceil_div(a.n, 128), 128, 0, s>>>(a, off);
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_energy(const EnergyArgs<real>& a, double* partial, int nblocks, double* out,
                          cudaStream_t s) {
  // at least four quads to a thread, where there are that many: a partial sum costs about as much
  const long long quads = (long long)a.B * a.Z * a.Y * (a.X / 4);
  nblocks = (int)std::min<long long>(nblocks, (quads + 4 * 256 - 1) / (4 * 256));
  energy_kernel<real><<<dim3(nblocks, 6), 256, 0, s>>>(a, partial);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  energy_final_kernel<<<1, 192, 0, s>>>(partial, nblocks, out);
  return cudaGetLastError();
}

template <typename real>
int dft_blocks(const ProbeArgs<real>& a, bool tail) {
  return dft_blocks_of(a, tail);
}

template <typename real>
cudaError_t launch_dft(const ProbeArgs<real>& a, int n, int kinds, bool tail, int bump, cudaStream_t s) {
  // tail: the direct sweeps' launches, all of which take part
  return launch_pdl(tail, dft_kernel<real>, dim3(dft_blocks_of(a, tail)), dim3(kDftF * kChunk), 0, s, a, n, kinds,
                    tail ? 1 : 0, bump);
}

template <typename real>
cudaError_t launch_dft_batch(const ProbeArgs<real>* A, const BatchGrid& G, int blocks, int n, bool tail,
                             cudaStream_t s) {
  if (blocks <= 0) return cudaSuccess;
  return launch_pdl(tail, dft_batch_kernel<real>, dim3(blocks), dim3(kDftF * kChunk), 0, s, A, G, n, tail ? 1 : 0);
}

#define OAFDTD_INSTANTIATE(real)                                                                   \
  template cudaError_t launch_ghosts<real>(real* const[3], int, int, int, int, int, int, int,      \
                                           cudaStream_t, bool);                                     \
  template cudaError_t launch_pre_e<real>(const ProbeArgs<real>&, int, cudaStream_t);              \
  template cudaError_t launch_probe_e<real>(const ProbeArgs<real>&, int, cudaStream_t);            \
  template cudaError_t launch_edges<real>(const EdgeArgs<real>&, int, cudaStream_t);               \
  template cudaError_t launch_sibc<real>(const SibcArgs<real>&, cudaStream_t, int, int, bool);      \
  template int dft_blocks<real>(const ProbeArgs<real>&, bool);                                      \
  template cudaError_t launch_dft<real>(const ProbeArgs<real>&, int, int, bool, int, cudaStream_t); \
  template cudaError_t launch_dft_batch<real>(const ProbeArgs<real>*, const BatchGrid&, int, int, bool, \
                                              cudaStream_t);                                        \
  template int pre_e_blocks<real>(const ProbeArgs<real>&);                                          \
  template int probe_e_blocks<real>(const ProbeArgs<real>&);                                        \
  template int edge_blocks<real>(const EdgeArgs<real>&);                                            \
  template int sibc_blocks<real>(const SibcArgs<real>&);                                            \
  template int sibc_variant<real>(const SibcArgs<real>&);                                           \
  template cudaError_t launch_pre_e_batch<real>(const ProbeArgs<real>*, const BatchGrid&, int, int, \
                                                cudaStream_t);                                      \
  template cudaError_t launch_probe_e_batch<real>(const ProbeArgs<real>*, const BatchGrid&, int, int, \
                                                  cudaStream_t);                                    \
  template cudaError_t launch_edges_batch<real>(const EdgeArgs<real>*, const BatchGrid&, int, int,  \
                                                cudaStream_t);                                      \
  template cudaError_t launch_sibc_batch<real>(const SibcArgs<real>*, const BatchGrid&, int, int, bool,   \
                                               cudaStream_t);                                       \
  template cudaError_t preload_kernels<real>();                                                     \
  template cudaError_t launch_energy<real>(const EnergyArgs<real>&, double*, int, double*,         \
                                           cudaStream_t);

template <typename real>
cudaError_t preload_kernels() {
  cudaFuncAttributes fa;
  const void* fns[] = {
      reinterpret_cast<const void*>(ghost_kernel<real>),
      reinterpret_cast<const void*>(pre_e_kernel<real>),
      reinterpret_cast<const void*>(probe_e_kernel<real>),
      reinterpret_cast<const void*>(sibc_kernel<real, 2, 16>),
      reinterpret_cast<const void*>(sibc_kernel<real, 1, 16>),
      reinterpret_cast<const void*>(sibc_kernel<real, 4, 16>),
      reinterpret_cast<const void*>(sibc_generic_kernel<real>),
      reinterpret_cast<const void*>(edge_kernel<real>),
      reinterpret_cast<const void*>(energy_kernel<real>),
      reinterpret_cast<const void*>(energy_final_kernel),
      reinterpret_cast<const void*>(dft_kernel<real>),
      reinterpret_cast<const void*>(dft_batch_kernel<real>),
      reinterpret_cast<const void*>(pre_e_batch_kernel<real>),
      reinterpret_cast<const void*>(probe_e_batch_kernel<real>),
      reinterpret_cast<const void*>(sibc_batch_kernel<real, 2, 16>),
      reinterpret_cast<const void*>(sibc_batch_kernel<real, 1, 16>),
      reinterpret_cast<const void*>(sibc_batch_kernel<real, 4, 16>),
      reinterpret_cast<const void*>(sibc_batch_kernel<real, 0, 16>),
      reinterpret_cast<const void*>(edge_batch_kernel<real>),
  };
  for (const void* f : fns) {
    const cudaError_t err = cudaFuncGetAttributes(&fa, f);
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

OAFDTD_INSTANTIATE(float)
OAFDTD_INSTANTIATE(double)

}  // namespace oafdtd
