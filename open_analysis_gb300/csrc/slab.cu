// The direct kernels: H and E updates read straight from global memory, no staging.
//
// The update domain of each sweep is split into an interior box, which holds no CPML correction
// cell and is swept by the staged or fused kernels (staged.cu, fused.cu), and up to six disjoint
// boxes around it: these kernels march those boxes. In variant 0 they have the whole domain, as one box
// in float32; it is the default of float64 grids and of float32 grids whose fields mostly stay in the
// L2 cache.
//
// Each thread owns one component of one 16-byte vector of x cells (four float32 or two float64) of one
// storage row and marches a few z planes, carrying the plane its z derivative needs again; the three
// components of a column sit in one block, so the sources they share are read once into its L1.
// Per plane every load is issued first (sources, field, index, Debye current, psi), then the
// arithmetic, then the stores, so no load waits behind a store it cannot be proven not to alias; and
// the next plane's lines are prefetched into L2, which needs no registers. What bounds these kernels
// is the latency of those loads at 24 warps per SM, which leaves a thread 80 registers (spilled bytes:
// H none; E in float32 40 with one pole, 136 with several, in float64 232 and 112; the batched kernels,
// whose arguments are in shared memory, H 8 and 32, E 236, 320, 292 and 308): at 400x400x120, batch 2, over the
// whole grid H takes 0.31 ms and E 0.49 ms (4.5 and 4.1 TB/s of the measured 6.8; 0.32 and 0.52
// without the prefetch at 16 planes). Three shapes measured and left: every component in one thread
// (168 registers, 0.62 and 1.53 ms), one plane per thread (set-up dominates: 0.59 and 0.88 ms), one
// body for all three components (600 instead of 300 instructions per vector in E).
//
// For every cell, in the reference's order (packages/oa-fdtd/src/oa_fdtd/reference.py:152-207,
// :115-127):
//   1. the bulk update (E: ca E + cb curl H; H: H + dt/mu0 curl E);
//   2. the CPML corrections of the component in ascending derivative axis, each
//      psi <- b psi + c d; F <- F + (sign k)(ek d + psi), with d the derivative the bulk update
//      used and k = cb of the edge (E) or dt/mu0 (H);
//   3. (E) the Debye update of dispersive edges: jt = 1/2 sum_p (1 + k_p) J_p;
//      E^{n+1} = E - cbe jt; J_p = k_p J_p + beta_p (E^{n+1} - E^n);
// In variant 0 the E launch also takes the edge list's edges (injection, and the Debye update of the
// dispersive ones): a few blocks of one thread per edge do their whole update, and the vector
// threads, which know those edges by table entries of their own past edge_lo, leave them out.
// Elsewhere the edge pass does this after the sweeps.
// The library is compiled without FMA contraction, so each product and sum rounds as in NumPy.
//
// psi layout, one array per (kind, component, axis, side): (B, Z', Y', X') with the slab width
// on the derivative axis and the full storage extent on the other two.

#include <algorithm>

#include "device_common.cuh"
#include "probe.cuh"

namespace oafdtd {

// A block: vector columns x 3 components (threadIdx.x, y).
constexpr int kSlabCols = 64, kSlabThreads = 3 * kSlabCols;

// One 16-byte vector of consecutive x cells: the cells a thread owns.
template <typename real>
struct Vec {
  static constexpr int n = 16 / (int)sizeof(real);
  real v[n];
};
template <typename real>
constexpr int kVec = Vec<real>::n;

__device__ __forceinline__ Vec<float> ldv(const float* p) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  return Vec<float>{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ Vec<double> ldv(const double* p) {
  const double2 t = *reinterpret_cast<const double2*>(p);
  return Vec<double>{{t.x, t.y}};
}
__device__ __forceinline__ void stv(float* p, const Vec<float>& q) {
  *reinterpret_cast<float4*>(p) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}
__device__ __forceinline__ void stv(double* p, const Vec<double>& q) {
  *reinterpret_cast<double2*>(p) = make_double2(q.v[0], q.v[1]);
}
// The material indices of one vector of cells, packed.
template <typename real>
struct Mats {
  uint32_t w[kVec<real> / 2];
  __device__ __forceinline__ int operator[](int e) const { return (int)((w[e / 2] >> (16 * (e & 1))) & 0xffffu); }
  __device__ __forceinline__ bool same() const {
    return w[0] == w[kVec<real> / 2 - 1] && (w[0] >> 16) == (w[0] & 0xffffu);
  }
};
__device__ __forceinline__ void ld_mat(const uint16_t* p, Mats<float>& m) {
  const uint2 t = *reinterpret_cast<const uint2*>(p);
  m.w[0] = t.x, m.w[1] = t.y;
}
__device__ __forceinline__ void ld_mat(const uint16_t* p, Mats<double>& m) { m.w[0] = *reinterpret_cast<const uint32_t*>(p); }
template <typename real>
__device__ __forceinline__ Vec<real> zerov() {
  Vec<real> z;
#pragma unroll
  for (int e = 0; e < kVec<real>; ++e) z.v[e] = (real)0;
  return z;
}

// n / f.d for n >= 0, by a multiplication where it is exact (the host sets m to 0 where it is not).
__device__ __forceinline__ int fast_div(const FastDiv& f, int n) {
  return f.m ? (int)__umulhi((unsigned)n, f.m) : n / f.d;
}

// Where a thread works: member, storage row, first cell of its vector, planes; core: its cells lie in
// no correction box.
struct SlabWork {
  int b, j, i0, k0, k1;
  bool live, core;
};

template <typename real>
__device__ __forceinline__ SlabWork slab_work(const SlabLaunch& L, int nx, int blk) {
  constexpr int V = kVec<real>;
  int s = 0;
  while (s + 1 < L.n && blk >= L.first[s + 1]) ++s;
  const Span3 bx = L.box[s];
  const int r = blk - L.first[s];
  // Member fastest: the members of a column block run side by side and read its indices, metrics and
  // CPML coefficients from memory once (120x60x40, two members: 21.5 to 20.0 us a step; the slabs' E of
  // 397x323x160, eight members: 503 to 476 us).
  SlabWork w;
  int t = r;
  w.b = 0;
  if (L.nb.d != 1) {
    t = fast_div(L.nb, r);
    w.b = r - t * L.nb.d;
  }
  const int ch = fast_div(L.cblk[s], t), cb = t - ch * L.cblk[s].d;
  const int c = cb * kSlabCols + (int)threadIdx.x;
  const int row = fast_div(L.nv[s], c);
  w.j = bx.j0 + row;
  w.i0 = 4 * bx.q0 + V * (c - row * L.nv[s].d);
  w.k0 = bx.k0 + ch * L.planes;
  w.k1 = min(w.k0 + L.planes, bx.k1);
  w.live = w.j < bx.j1 && w.i0 <= nx + 1;
  const Span3& o = L.core;
  w.core = w.i0 >= 4 * o.q0 && w.i0 + V <= 4 * o.q1 && w.j >= o.j0 && w.j < o.j1 && w.k0 >= o.k0 && w.k1 <= o.k1;
  return w;
}

// The cells of a vector from i0 on that lie in 1 .. last, one bit each.
template <typename real>
__device__ __forceinline__ unsigned valid_cells(int i0, int last) {
  constexpr int V = kVec<real>;
  const int n = last - i0 + 1;  // cells up to the last
  unsigned m = n >= V ? (1u << V) - 1u : (1u << n) - 1u;
  return i0 == 0 ? m & ~1u : m;
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

// ------------------------------------------------------------------------------------- CPML
// One correction term of a component (AX: its derivative axis) on a thread's column, worked out once
// for the march: psi of the march's first plane is at p, of the next a stride further on; `mask` holds
// the vector's cells inside the box (low bits) and, from bit 8, the march's planes inside it (0: no
// slab of this term holds the column). A march meets at most one side of an axis in y, and in z
// (slab_plan sees to it); in x, where the two slabs of a very thin grid can share a vector, the kernels
// of such grids (kThin) keep a second column. y and z slabs keep psi rows at the field pitch, so their
// vectors are whole 16 bytes (elements outside the box are written back unchanged); x slabs are read
// per element.
template <typename real>
struct PsiCol {
  real* p;
  int stride;
  unsigned mask;
};

// The first side from `from` on that holds the column; returns the one after it.
template <typename real, int AX>
__device__ __forceinline__ int psi_column(const CpmlTerm<real>& T, PsiCol<real>& c, const SlabWork& w, int X, int Y,
                                          int Z, int from = 0) {
  constexpr int V = kVec<real>;
  c.mask = 0;
  c.p = nullptr;
  c.stride = 0;
  if (w.core) return 2;
#pragma unroll 1
  for (int sd = from; sd < 2; ++sd) {
    const CpmlSide<real>& s = T.side[sd];
    if (s.psi == nullptr || w.i0 + V <= s.lo[0] || w.i0 >= s.hi[0] || w.j < s.lo[1] || w.j >= s.hi[1] ||
        w.k1 <= s.lo[2] || w.k0 >= s.hi[2])
      continue;
    const int wd = s.hi[AX] - s.lo[AX];
    c.stride = AX == 0 ? Y * wd : (AX == 1 ? wd * X : Y * X);
    c.p = AX == 0   ? s.psi + (((long long)w.b * Z + w.k0) * Y + w.j) * wd + (w.i0 - s.lo[0])
          : AX == 1 ? s.psi + (((long long)w.b * Z + w.k0) * wd + (w.j - s.lo[1])) * X + w.i0
                    : s.psi + (((long long)w.b * wd + w.k0 - s.lo[2]) * Y + w.j) * X + w.i0;
    const int lo = max(s.lo[0] - w.i0, 0), hi = min(s.hi[0] - w.i0, V);
    const int klo = max(s.lo[2] - w.k0, 0), khi = min(s.hi[2], w.k1) - w.k0;
    c.mask = (((1u << hi) - 1u) & ~((1u << lo) - 1u)) | ((((1u << khi) - 1u) & ~((1u << klo) - 1u)) << 8);
    return sd + 1;
  }
  return 2;
}

// psi of plane t of the march (false: the plane has none of this term); the march moves p on by the
// stride after each plane.
template <typename real, int AX>
__device__ __forceinline__ bool psi_load(const PsiCol<real>& c, Vec<real>& v, int t) {
  if (!((c.mask >> (8 + t)) & 1)) return false;
  if constexpr (AX == 0) {
#pragma unroll
    for (int e = 0; e < kVec<real>; ++e) v.v[e] = ((c.mask >> e) & 1) ? c.p[e] : (real)0;
  } else {
    v = ldv(c.p);
  }
  return true;
}

// psi <- b psi + c d; F <- F + (sign k)(ek d + psi) for the cells of the box, kf(e) the factor k of
// cell e; the updated psi back. The coefficient arrays are read-only for the whole run.
template <typename real, int AX, typename KF>
__device__ __forceinline__ void psi_apply(const PsiCol<real>& c, Vec<real>& v, const real* const (&co)[3], real sign,
                                          Vec<real>& f, const Vec<real>& d, KF kf, const SlabWork& w, int k) {
  Vec<real> cb, cc, ck;
  if constexpr (AX == 0) {
    cb = ldv(co[0] + w.i0), cc = ldv(co[1] + w.i0), ck = ldv(co[2] + w.i0);
  } else {
    const int ia = AX == 1 ? w.j : k;
    const real b = __ldg(co[0] + ia), cv = __ldg(co[1] + ia), kv = __ldg(co[2] + ia);
#pragma unroll
    for (int e = 0; e < kVec<real>; ++e) cb.v[e] = b, cc.v[e] = cv, ck.v[e] = kv;
  }
#pragma unroll
  for (int e = 0; e < kVec<real>; ++e) {
    if (!((c.mask >> e) & 1)) continue;
    real ps = v.v[e] * cb.v[e];
    ps = ps + cc.v[e] * d.v[e];
    v.v[e] = ps;
    const real upd = ck.v[e] * d.v[e] + ps;
    f.v[e] = f.v[e] + (sign * kf(e)) * upd;
  }
  if constexpr (AX == 0) {
#pragma unroll
    for (int e = 0; e < kVec<real>; ++e)
      if ((c.mask >> e) & 1) c.p[e] = v.v[e];
  } else {
    stv(c.p, v);
  }
}

// ------------------------------------------------------------------------------------- E
// One edge of the edge list for one member, whole: bulk update, injection (reference.py:223-234),
// Debye update. The vector threads leave these edges (and their currents) alone, so nothing else
// writes them; the host keeps edges in CPML boxes and on copper to the edge pass.
template <typename real>
__device__ __forceinline__ void list_edge(const SweepArgs<real>& a, const EdgeArgs<real>& ed, int off, int t) {
  const int n = t % ed.n, b = t / ed.n;
  const int c = ed.comp[n], X = a.X;
  const int q = (int)ed.flat[n], sz = X * a.Y;
  const int k = q / sz, j = (q - k * sz) / X, i = q - k * sz - j * X;
  const long long base = (long long)b * a.bs;
  const real* Hx = a.Ho[0] + base + q;
  const real* Hy = a.Ho[1] + base + q;
  const real* Hz = a.Ho[2] + base + q;
  const int m = a.mat[c][q];
  const Coef<real> cf = ldg_coef(a.coef + m);
  const real e0 = a.E[c][base + q];
  real val = e0;
  if (i >= 1 && i <= a.nx + 1 && j >= 1 && j <= a.ny + 1 && k >= 1 && k <= a.nz + 1) {
    real d0, d1;
    if (c == 0) {
      d0 = (Hz[0] - Hz[-X]) * a.idd[1][j];
      d1 = (Hy[0] - Hy[-sz]) * a.idd[2][k];
    } else if (c == 1) {
      d0 = (Hz[0] - Hz[-1]) * a.idd[0][i];
      d1 = (Hx[0] - Hx[-sz]) * a.idd[2][k];
    } else {
      d0 = (Hy[0] - Hy[-1]) * a.idd[0][i];
      d1 = (Hx[0] - Hx[-X]) * a.idd[1][j];
    }
    const real acc = c != 1 ? d0 + (-d1) : d1 + (-d0);
    val = cf.ca * val + cf.cb * acc;
  }
  const long long step = *ed.step_base + off;
  const int ie = ed.inj_end[n];
#pragma unroll 1
  for (int s = ed.inj_beg[n]; s < ie; ++s) {
    const int ch = ed.i_chan[s];
    const double w = ed.wave[(long long)ch * ed.max_steps + step];
    val = val + (real)((ed.drive[b * ed.n_chan + ch] * w) * ed.i_amp[s]);
  }
  if (ed.def_slot[n] >= 0) {
    const int P = a.ade_P;
    const long long js = (long long)a.B * a.jnk[c] * sz;
    real* J = a.J[c] + ((long long)b * a.jnk[c] - a.jk0[c]) * sz + q;
    real jt = (real)0;
#pragma unroll 1
    for (int p = 0; p < P; ++p) jt = jt + a.ade_onekp[p] * J[p * js];
    jt = (real)0.5 * jt;
    const real en = val - cf.cbe * jt;
    const real de = en - e0;
#pragma unroll 1
    for (int p = 0; p < P; ++p) {
      const real bp = p == 0 ? cf.beta0 : a.ade_beta[(long long)m * P + p];
      J[p * js] = a.ade_kp[p] * J[p * js] + bp * de;
    }
    val = en;
  }
  a.Eo[c][base + q] = val;
}

// Stores a vector; the elements of the edge list's edges stay out (listed: there are some).
template <typename real>
__device__ __forceinline__ void st_unlisted(real* p, const Vec<real>& v, const Mats<real>& m, int edge_lo, bool listed) {
  if (!listed) {
    stv(p, v);
  } else {
#pragma unroll
    for (int e = 0; e < kVec<real>; ++e)
      if (m[e] < edge_lo) p[e] = v.v[e];
  }
}

// One E component on one vector column. Per plane every load first (H, E, indices, Debye current,
// psi), then the arithmetic, then every store. C: 0 Ex (terms y +Hz, z -Hy), 1 Ey (z +Hx, x -Hz),
// 2 Ez (x +Hy, y -Hx). kMulti: more than one Debye pole; the currents of each pole are then read
// twice (the second time from the L1 cache). kThin: a vector may lie in both x slabs (slab_thin).
template <typename real, int C, bool kMulti, bool kThin>
__device__ __forceinline__ void slab_e_march(const SweepArgs<real>& a, bool inject, const SlabWork& w) {
  constexpr int V = kVec<real>;
  constexpr int A0 = C == 0 ? 1 : 0, A1 = C == 2 ? 1 : 2;  // the derivative axes, ascending
  // Vectors whose cells have several table entries: a branch of their own in float32 (one gather and
  // four registers serve the rest); in float64 both branches would issue their arithmetic wherever
  // a warp holds both, and the two float64 operations a clock and SM bound the kernel (0.51 against
  // 0.46 ms for E at 161x143x88, batch 2): there every cell has its entry.
  constexpr bool kBranch = sizeof(real) == 4;
  const int X = a.X, Y = a.Y, i0 = w.i0, sz = X * Y;
  const long long base = (long long)w.b * a.bs;
  const real* const s0 = a.Ho[C == 2 ? 1 : 2] + base;  // sources along A0 and A1: H^{n+1/2}
  const real* const s1 = a.Ho[C == 0 ? 1 : 0] + base;
  const real* const E = a.E[C] + base;                 // E^n
  real* const Eo = a.Eo[C] + base;                     // E^{n+1}
  real* const J = a.J[C] + (long long)(w.b * a.jnk[C] - a.jk0[C]) * sz;
  const int jlo = a.ade_P > 0 ? a.jk0[C] : 1 << 30, jhi = a.jk0[C] + a.jnk[C];
  const uint16_t* const mat = a.mat[C];
  Vec<real> wx;
  if (C != 0) wx = ldv(a.idd[0] + i0);
  const real wy = a.idd[1][w.j];
  const unsigned vm = valid_cells<real>(i0, a.nx + 1);
  PsiCol<real> c0, c1, c2{};  // c2: the other x slab
  const int other = psi_column<real, A0>(a.ecorr[C][0], c0, w, X, Y, a.nz + 2);
  if (kThin && A0 == 0) psi_column<real, A0>(a.ecorr[C][0], c2, w, X, Y, a.nz + 2, other);
  psi_column<real, A1>(a.ecorr[C][1], c1, w, X, Y, a.nz + 2);
  int q = (w.k0 * Y + w.j) * X + i0;  // offset within one member (below 2^31)
  Vec<real> below;                    // the z-derivative's source on the plane below, carried
  if (C != 2) below = ldv(s1 + (q - sz));
#pragma unroll 1
  for (int k = w.k0; k < w.k1; ++k, q += sz, c0.p += c0.stride, c1.p += c1.stride, c2.p += c2.stride) {
    // ---- loads
    Mats<real> m;
    ld_mat(mat + q, m);
    const Vec<real> e0 = ldv(E + q);
    const Vec<real> u0 = ldv(s0 + q), u1 = ldv(s1 + q);
    Vec<real> n0, n1;      // the neighbours one down along A0 (y) and A1 (y); z is carried
    real x0 = (real)0;     // along x only element 0's; cell 0 is never updated: none from the row before
    if (C == 0) n0 = ldv(s0 + (q - X));
    else if (i0 > 0) x0 = s0[q - 1];
    if (C == 2) n1 = ldv(s1 + (q - X));
    else n1 = below;
    Vec<real> j4, p0, p1, p2;
    const bool debye = k >= jlo && k < jhi;
    if (!kMulti && debye) j4 = ldv(J + q);
    const bool on0 = psi_load<real, A0>(c0, p0, k - w.k0), on1 = psi_load<real, A1>(c1, p1, k - w.k0);
    const bool on2 = kThin && A0 == 0 && psi_load<real, A0>(c2, p2, k - w.k0);
    const real w1 = C == 2 ? wy : a.idd[2][k];
    if (k + 1 < w.k1) {
      prefetch_l2(mat + (q + sz));
      prefetch_l2(E + (q + sz));
      prefetch_l2(s0 + (q + sz));
      prefetch_l2(s1 + (q + sz));
      if (k + 1 >= jlo && k + 1 < jhi) prefetch_l2(J + (q + sz));
    }
    if (C != 2) below = u1;
    // ---- bulk update: d0 along A0, d1 along A1. The cells of a vector mostly share a table entry: one
    // gather then serves all of them
    Vec<real> d0, d1, f = e0;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      d0.v[e] = C == 0 ? (u0.v[e] - n0.v[e]) * wy : (u0.v[e] - (e > 0 ? u0.v[e > 0 ? e - 1 : 0] : x0)) * wx.v[e];
      d1.v[e] = (u1.v[e] - n1.v[e]) * w1;
    }
    auto acc = [&](int e) { return C != 1 ? d0.v[e] + (-d1.v[e]) : d1.v[e] + (-d0.v[e]); };
    const int m0 = m[0];
    const Coef<real> cf0 = ldg_coef(a.coef + m0);
    const bool same = m.same();
    unsigned dis = m0 >= a.ade_lo && m0 < a.ade_hi ? vm : 0u;
    bool listed = m0 >= a.edge_lo;
    Coef<real> cfd[kBranch ? 1 : V];
    if constexpr (!kBranch) {
      cfd[0] = cf0;
#pragma unroll
      for (int e = 1; e < V; ++e) {
        cfd[e] = cf0;
        if (m[e] != m0) cfd[e] = ldg_coef(a.coef + m[e]);
      }
    }
    auto coef = [&](int e) {
      if constexpr (!kBranch) return cfd[e];
      else return same ? cf0 : ldg_coef(a.coef + m[e]);
    };
    if (same || !kBranch) {
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const Coef<real> cf = kBranch ? cf0 : cfd[kBranch ? 0 : e];
        if ((vm >> e) & 1) f.v[e] = cf.ca * f.v[e] + cf.cb * acc(e);
      }
    }
    if (!same) {
      dis = 0;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        if constexpr (kBranch) {
          const Coef<real> cf = ldg_coef(a.coef + m[e]);
          if ((vm >> e) & 1) f.v[e] = cf.ca * f.v[e] + cf.cb * acc(e);
        }
        if (m[e] >= a.ade_lo && m[e] < a.ade_hi) dis |= vm & (1u << e);
        listed |= m[e] >= a.edge_lo;
      }
    }
    listed = listed && inject;
    // ---- corrections
    auto kf = [&](int e) { return coef(e).cb; };
    if (on0) psi_apply<real, A0>(c0, p0, a.pe[A0], a.ecorr[C][0].sign, f, d0, kf, w, k);
    if (on2) psi_apply<real, A0>(c2, p2, a.pe[A0], a.ecorr[C][0].sign, f, d0, kf, w, k);
    if (on1) psi_apply<real, A1>(c1, p1, a.pe[A1], a.ecorr[C][1].sign, f, d1, kf, w, k);
    // ---- Debye
    if (dis) {
      if constexpr (!kMulti) {
        const real onekp = a.ade_onekp[0], kp = a.ade_kp[0];
#pragma unroll
        for (int e = 0; e < V; ++e) {
          if (!((dis >> e) & 1)) continue;
          const Coef<real> cf = coef(e);
          const real jt = (real)0.5 * (onekp * j4.v[e]);
          const real en = f.v[e] - cf.cbe * jt;
          const real de = en - e0.v[e];
          j4.v[e] = kp * j4.v[e] + cf.beta0 * de;
          f.v[e] = en;
        }
        st_unlisted<real>(J + q, j4, m, a.edge_lo, listed);
      } else {
        const long long js = (long long)a.B * a.jnk[C] * sz;
        const int P = a.ade_P;
        Vec<real> jt = zerov<real>(), de;
#pragma unroll 4
        for (int p = 0; p < P; ++p) {
          const Vec<real> jp = ldv(J + q + p * js);
          const real onekp = a.ade_onekp[p];
#pragma unroll
          for (int e = 0; e < V; ++e) jt.v[e] = jt.v[e] + onekp * jp.v[e];
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const real en = f.v[e] - coef(e).cbe * ((real)0.5 * jt.v[e]);
          de.v[e] = en - e0.v[e];
          if ((dis >> e) & 1) f.v[e] = en;
        }
#pragma unroll 2
        for (int p = 0; p < P; ++p) {
          Vec<real> jp = ldv(J + q + p * js);
          const real kp = a.ade_kp[p], b0 = __ldg(a.ade_beta + m0 * P + p);
#pragma unroll
          for (int e = 0; e < V; ++e) {
            real bp = b0;
            if (e > 0 && m[e] != m0) bp = __ldg(a.ade_beta + m[e] * P + p);
            if ((dis >> e) & 1) jp.v[e] = kp * jp.v[e] + bp * de.v[e];
          }
          st_unlisted<real>(J + q + p * js, jp, m, a.edge_lo, listed);
        }
      }
    }
    st_unlisted<real>(Eo + q, f, m, a.edge_lo, listed);
  }
}

// The E boxes; the first L.extra blocks sample the H probes of the step instead (H is complete), the
// next L.inject blocks take the edge list's edges.
template <typename real, bool kMulti, bool kThin>
__device__ __forceinline__ void slab_e_body(const SweepArgs<real>& a, const SlabLaunch& L, const EdgeArgs<real>& ed,
                                            const ProbeArgs<real>& pr, int off, int block) {
  if (block < L.extra) {
    pdl_wait();
    probe_sample(pr, 1, block, off);
    return;
  }
  block -= L.extra;
  if (block < L.inject) {
    pdl_wait();
    const int t = block * kSlabThreads + (int)(threadIdx.x + kSlabCols * threadIdx.y);
    if (t < ed.n * a.B) list_edge<real>(a, ed, off, t);
    return;
  }
  const SlabWork w = slab_work<real>(L, a.nx, block - L.inject);
  pdl_wait();
  if (!w.live) return;
  const bool inject = L.inject > 0;
  if (threadIdx.y == 0) slab_e_march<real, 0, kMulti, kThin>(a, inject, w);
  else if (threadIdx.y == 1) slab_e_march<real, 1, kMulti, kThin>(a, inject, w);
  else slab_e_march<real, 2, kMulti, kThin>(a, inject, w);
}

template <typename real, bool kMulti, bool kThin>
__global__ void __launch_bounds__(kSlabThreads, 4)
    slab_e_kernel(const __grid_constant__ SweepArgs<real> a, const __grid_constant__ SlabLaunch L,
                  const __grid_constant__ EdgeArgs<real> ed, const __grid_constant__ ProbeArgs<real> pr, int off) {
  slab_e_body<real, kMulti, kThin>(a, L, ed, pr, off, (int)blockIdx.x);
}

// Several engines' E updates in one launch: engine e's arguments at A[e], L[e], ED[e] and PR[e].
template <typename real, bool kMulti, bool kThin>
__global__ void __launch_bounds__(kSlabThreads, 4)
    slab_e_batch_kernel(const SweepArgs<real>* __restrict__ A, const SlabLaunch* __restrict__ L,
                        const EdgeArgs<real>* __restrict__ ED, const ProbeArgs<real>* __restrict__ PR, const BatchGrid G,
                        int off) {
  __shared__ __align__(16) unsigned char args[sizeof(SweepArgs<real>)];
  __shared__ __align__(16) unsigned char launch[sizeof(SlabLaunch)];
  int e;
  const uint3 bid = G.block(&e);
  const SlabLaunch& l = stage_args(L + e, launch);
  slab_e_body<real, kMulti, kThin>(stage_args(A + e, args), l, ED[e], PR[e], off, (int)bid.x);
}

// ------------------------------------------------------------------------------------- H
// One H component on one vector column. C: 0 Hx (terms y -Ez, z +Ey), 1 Hy (z -Ex, x +Ez), 2 Hz
// (x -Ey, y +Ex). The cells each updates: Hx i in 1..nx+1, j <= ny, k <= nz; Hy i <= nx, k <= nz; Hz
// i <= nx, j <= ny. kThin as in slab_e_march.
template <typename real, int C, bool kThin>
__device__ __forceinline__ void slab_h_march(const SweepArgs<real>& a, const SlabWork& w) {
  constexpr int V = kVec<real>;
  constexpr int A0 = C == 0 ? 1 : 0, A1 = C == 2 ? 1 : 2;  // the derivative axes, ascending
  if (C != 1 && w.j > a.ny) return;
  const int k1 = C == 2 ? w.k1 : min(w.k1, a.nz + 1);
  const int X = a.X, Y = a.Y, i0 = w.i0, sz = X * Y;
  const long long base = (long long)w.b * a.bs;
  const real* const s0 = a.E[C == 2 ? 1 : 2] + base;  // sources along A0 and A1
  const real* const s1 = a.E[C == 0 ? 1 : 0] + base;
  const real* const H = a.H[C] + base;                // H^{n-1/2}
  real* const Ho = a.Ho[C] + base;                    // H^{n+1/2}
  Vec<real> wx;
  if (C != 0) wx = ldv(a.ip[0] + i0);
  const real wy = a.ip[1][w.j];
  const bool right = i0 + V < X;  // the x + 1 neighbour of the last element is in the row
  const unsigned vm = valid_cells<real>(i0, C == 0 ? a.nx + 1 : a.nx);
  const real dtmu = a.dtmu;
  PsiCol<real> c0, c1, c2{};  // c2: the other x slab
  const int other = psi_column<real, A0>(a.hcorr[C][0], c0, w, X, Y, a.nz + 2);
  if (kThin && A0 == 0) psi_column<real, A0>(a.hcorr[C][0], c2, w, X, Y, a.nz + 2, other);
  psi_column<real, A1>(a.hcorr[C][1], c1, w, X, Y, a.nz + 2);
  int q = (w.k0 * Y + w.j) * X + i0;
  Vec<real> here;  // the z-derivative's source on this plane, carried from the last one's plane above
  if (C != 2) here = ldv(s1 + q);
#pragma unroll 1
  for (int k = w.k0; k < k1; ++k, q += sz, c0.p += c0.stride, c1.p += c1.stride, c2.p += c2.stride) {
    // ---- loads
    Vec<real> h = ldv(H + q);
    const Vec<real> u0 = ldv(s0 + q);
    Vec<real> n0, u1, n1;  // the neighbours one up along A0 (y) and A1 (z, y)
    real x0 = (real)0;     // along x only the last element's
    if (C == 0) n0 = ldv(s0 + (q + X));
    else if (right) x0 = s0[q + V];
    if (C == 2) {
      u1 = ldv(s1 + q);
      n1 = ldv(s1 + (q + X));
    } else {
      u1 = here;
      n1 = ldv(s1 + (q + sz));
      here = n1;
    }
    Vec<real> p0, p1, p2;
    const bool on0 = psi_load<real, A0>(c0, p0, k - w.k0), on1 = psi_load<real, A1>(c1, p1, k - w.k0);
    const bool on2 = kThin && A0 == 0 && psi_load<real, A0>(c2, p2, k - w.k0);
    const real w1 = C == 2 ? wy : a.ip[2][k];
    if (k + 1 < k1) {
      prefetch_l2(H + (q + sz));
      prefetch_l2(s0 + (q + sz));
      if (C == 2) prefetch_l2(s1 + (q + sz));
      else if (k + 2 < a.nz + 2) prefetch_l2(s1 + (q + 2 * sz));
    }
    // ---- arithmetic: d0 along A0, d1 along A1
    Vec<real> d0, d1;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      d0.v[e] = C == 0 ? (n0.v[e] - u0.v[e]) * wy
                       : ((e < V - 1 ? u0.v[e < V - 1 ? e + 1 : e] : x0) - u0.v[e]) * wx.v[e];
      d1.v[e] = (n1.v[e] - u1.v[e]) * w1;
      const real acc = C == 1 ? (-d1.v[e]) + d0.v[e] : (-d0.v[e]) + d1.v[e];
      if ((vm >> e) & 1) h.v[e] = h.v[e] + dtmu * acc;
    }
    auto kf = [&](int) { return dtmu; };
    if (on0) psi_apply<real, A0>(c0, p0, a.ph[A0], a.hcorr[C][0].sign, h, d0, kf, w, k);
    if (on2) psi_apply<real, A0>(c2, p2, a.ph[A0], a.hcorr[C][0].sign, h, d0, kf, w, k);
    if (on1) psi_apply<real, A1>(c1, p1, a.ph[A1], a.hcorr[C][1].sign, h, d1, kf, w, k);
    stv(Ho + q, h);
  }
}

template <typename real, bool kThin>
__device__ __forceinline__ void slab_h_body(const SweepArgs<real>& a, const SlabLaunch& L, int block) {
  const SlabWork w = slab_work<real>(L, a.nx, block);
  pdl_wait();
  if (!w.live) return;
  if (threadIdx.y == 0) slab_h_march<real, 0, kThin>(a, w);
  else if (threadIdx.y == 1) slab_h_march<real, 1, kThin>(a, w);
  else slab_h_march<real, 2, kThin>(a, w);
}

// The H boxes; the first L.extra blocks sample the E probes of the previous step instead (the H
// update leaves E alone; off - 1 is that step).
template <typename real, bool kThin>
__global__ void __launch_bounds__(kSlabThreads, 4)
    slab_h_kernel(const __grid_constant__ SweepArgs<real> a, const __grid_constant__ SlabLaunch L,
                  const __grid_constant__ ProbeArgs<real> pr, int off) {
  if ((int)blockIdx.x < L.extra) {
    pdl_wait();
    probe_sample(pr, 0, (int)blockIdx.x, off - 1);
    return;
  }
  slab_h_body<real, kThin>(a, L, (int)blockIdx.x - L.extra);
}

// Several engines' H updates in one launch. The E probes of a step before the first of a group
// (off 0) are already in: those blocks return.
template <typename real, bool kThin>
__global__ void __launch_bounds__(kSlabThreads, 4)
    slab_h_batch_kernel(const SweepArgs<real>* __restrict__ A, const SlabLaunch* __restrict__ L,
                        const ProbeArgs<real>* __restrict__ PR, const BatchGrid G, int off) {
  __shared__ __align__(16) unsigned char args[sizeof(SweepArgs<real>)];
  __shared__ __align__(16) unsigned char launch[sizeof(SlabLaunch)];
  int e;
  const uint3 bid = G.block(&e);
  const SlabLaunch& l = stage_args(L + e, launch);
  if ((int)bid.x < l.extra) {
    pdl_wait();
    if (off > 0) probe_sample(PR[e], 0, (int)bid.x, off - 1);
    return;
  }
  slab_h_body<real, kThin>(stage_args(A + e, args), l, (int)bid.x - l.extra);
}

// ------------------------------------------------------------------------------------- launch
// The divisor d for operands below `limit`: ceil(2^32 / d) divides exactly by the high half of a
// multiplication where limit * (its excess over 2^32) stays below 2^32.
static FastDiv fast_divisor(long long d, long long limit) {
  FastDiv f{(int)d, 0};
  const unsigned long long m = ((1ull << 32) + (unsigned long long)d - 1) / (unsigned long long)d;
  const unsigned long long excess = m * (unsigned long long)d - (1ull << 32);
  if (d > 1 && (unsigned long long)limit * std::max(excess, 1ull) < (1ull << 32)) f.m = (unsigned)m;
  return f;
}

// Whether a vector of cells can lie in both x slabs of a term (grids of twice the slab and a cell or
// two): the kernels then keep a second x column, which takes registers that the others need.
template <typename real>
bool slab_thin(const SweepArgs<real>& a, int kind) {
  constexpr int V = kVec<real>;
  for (int c = 1; c < 3; ++c) {
    const CpmlTerm<real>& T = kind == 0 ? a.ecorr[c][0] : a.hcorr[c][0];
    const CpmlSide<real>* s = T.side;
    if (s[0].psi == nullptr || s[1].psi == nullptr) continue;
    const int lo = s[0].lo[0] < s[1].lo[0] ? 0 : 1;
    if ((s[lo].hi[0] - 1) / V >= s[1 - lo].lo[0] / V) return true;
  }
  return false;
}

// Vectors of the boxes of one kind, all members.
template <typename real>
long long slab_vecs(const SweepArgs<real>& a, int kind) {
  long long n = 0;
  for (int s = 0; s < a.n_slab[kind]; ++s) {
    const Span3& bx = a.slab[kind][s];
    const long long q = std::min(bx.q1, (a.nx + 1) / 4 + 1) - bx.q0;
    if (q > 0 && bx.j1 > bx.j0 && bx.k1 > bx.k0) n += q * (4 / kVec<real>)*(bx.j1 - bx.j0) * (bx.k1 - bx.k0) * a.B;
  }
  return n;
}

// Planes a thread marches in a launch over `vecs` vectors. A thread's set-up (its place, the CPML
// columns) costs about one plane's work, so long marches pay as long as the blocks still fill the
// chip: 4 blocks of 192 threads per SM, 608 of them, run at once. us per step by planes (1, 2, 4, 8,
// 16), both sweeps over the whole grid: 6.7 thousand vectors 11 / 12 / 15 / 22 / 35; 155 thousand
// 28 / 23 / 22 / 26 / 39; 510 thousand 93 / 76 / 71 / 71 / 80; 1.2 million 224 / 182 / 159 / 150 /
// 154; 9.9 million 1632 / 1234 / 1013 / 920 / 886; a batch of 16 instances, 4.9 million together,
// 1138 / 812 / 642 / 552 / 521.
int slab_planes(long long vecs) {
  const long long blocks = vecs / kSlabCols;  // with one plane each
  return blocks >= 16 * 2400 ? 16 : (blocks >= 8 * 900 ? 8 : (blocks >= 4 * 600 ? 4 : (blocks >= 2 * 600 ? 2 : 1)));
}

template <typename real>
cudaError_t slab_plan(const SweepArgs<real>& a, int kind, SlabLaunch* L, long long* blocks, int planes) {
  *L = SlabLaunch{};
  *blocks = 0;
  L->core = a.core[kind];
  L->planes = planes > 0 ? planes : slab_planes(slab_vecs(a, kind));
  // no march may meet both z slabs of a term (a thread keeps one side's psi)
  for (int c = 0; c < 3; ++c)
    for (int t = 0; t < 2; ++t) {
      const CpmlTerm<real>& T = kind == 0 ? a.ecorr[c][t] : a.hcorr[c][t];
      if (T.axis != 2 || T.side[0].psi == nullptr || T.side[1].psi == nullptr) continue;
      const int gap = std::max(T.side[1].lo[2] - T.side[0].hi[2], T.side[0].lo[2] - T.side[1].hi[2]);
      L->planes = std::max(1, std::min(L->planes, gap + 1));
    }
  constexpr int kPerQuad = 4 / kVec<real>;
  long long total = 0;
  for (int n = 0; n < a.n_slab[kind]; ++n) {
    Span3 bx = a.slab[kind][n];
    bx.q1 = std::min(bx.q1, (a.nx + 1) / 4 + 1);  // quads past the last updated cell hold no work
    const long long cols = (long long)(bx.q1 - bx.q0) * kPerQuad * (bx.j1 - bx.j0);
    if (cols <= 0 || bx.k1 <= bx.k0) continue;
    L->box[L->n] = bx;
    L->first[L->n] = (int)total;
    const long long cblk = (cols + kSlabCols - 1) / kSlabCols;
    const int nch = (bx.k1 - bx.k0 + L->planes - 1) / L->planes;
    const long long blocks_here = cblk * nch * a.B;
    L->cblk[L->n] = fast_divisor(cblk, cblk * nch);
    L->nv[L->n] = fast_divisor((bx.q1 - bx.q0) * kPerQuad, cblk * kSlabCols);
    total += blocks_here;
    ++L->n;
  }
  if (total > 2147483647LL) return cudaErrorInvalidConfiguration;
  L->first[L->n] = (int)total;
  L->nb = fast_divisor(a.B, total);
  *blocks = total;
  return cudaSuccess;
}

template <typename real>
int inject_blocks(const EdgeArgs<real>& ed) {
  return (int)(((long long)ed.n * ed.B + kSlabThreads - 1) / kSlabThreads);
}

template <typename real>
cudaError_t launch_slab(const SweepArgs<real>& a, int kind, cudaStream_t s, const EdgeArgs<real>* ed,
                        const ProbeArgs<real>* pr, int off, bool pdl) {
  SlabLaunch L;
  long long blocks = 0;
  if (const cudaError_t e = slab_plan(a, kind, &L, &blocks)) return e;
  if (pr != nullptr) L.extra = kind == 0 ? pr->n_kind[1] * a.B : (off > 0 ? pr->n_kind[0] * a.B : 0);
  if (ed != nullptr) L.inject = inject_blocks(*ed);
  blocks += L.extra + L.inject;
  if (blocks == 0) return cudaSuccess;
  const EdgeArgs<real> no_ed{};
  const ProbeArgs<real> no_pr{};
  const EdgeArgs<real>& e = ed ? *ed : no_ed;
  const ProbeArgs<real>& p = pr ? *pr : no_pr;
  const dim3 grid((unsigned)blocks), block(kSlabCols, 3);
  const bool thin = slab_thin(a, kind);
  if (kind == 1)
    return launch_pdl(pdl, thin ? slab_h_kernel<real, true> : slab_h_kernel<real, false>, grid, block, 0, s, a, L, p,
                      off);
  auto kernel = a.ade_P > 1 ? (thin ? slab_e_kernel<real, true, true> : slab_e_kernel<real, true, false>)
                            : (thin ? slab_e_kernel<real, false, true> : slab_e_kernel<real, false, false>);
  return launch_pdl(pdl, kernel, grid, block, 0, s, a, L, e, p, off);
}

template <typename real>
cudaError_t launch_slab_batch(const SweepArgs<real>* A, const SlabLaunch* L, const EdgeArgs<real>* ED,
                              const ProbeArgs<real>* PR, const BatchGrid& G, int blocks, int kind, bool multi_pole,
                              bool thin, int off, bool pdl, cudaStream_t s) {
  if (blocks <= 0) return cudaSuccess;
  const dim3 grid(blocks), block(kSlabCols, 3);
  if (kind == 1)
    return launch_pdl(pdl, thin ? slab_h_batch_kernel<real, true> : slab_h_batch_kernel<real, false>, grid, block, 0, s,
                      A, L, PR, G, off);
  auto kernel = multi_pole ? (thin ? slab_e_batch_kernel<real, true, true> : slab_e_batch_kernel<real, true, false>)
                           : (thin ? slab_e_batch_kernel<real, false, true> : slab_e_batch_kernel<real, false, false>);
  return launch_pdl(pdl, kernel, grid, block, 0, s, A, L, ED, PR, G, off);
}

template <typename real>
cudaError_t preload_slab() {
  cudaFuncAttributes fa;
  const void* fns[] = {
      reinterpret_cast<const void*>(slab_e_kernel<real, false, false>),
      reinterpret_cast<const void*>(slab_e_kernel<real, false, true>),
      reinterpret_cast<const void*>(slab_e_kernel<real, true, false>),
      reinterpret_cast<const void*>(slab_e_kernel<real, true, true>),
      reinterpret_cast<const void*>(slab_h_kernel<real, false>),
      reinterpret_cast<const void*>(slab_h_kernel<real, true>),
      reinterpret_cast<const void*>(slab_e_batch_kernel<real, false, false>),
      reinterpret_cast<const void*>(slab_e_batch_kernel<real, false, true>),
      reinterpret_cast<const void*>(slab_e_batch_kernel<real, true, false>),
      reinterpret_cast<const void*>(slab_e_batch_kernel<real, true, true>),
      reinterpret_cast<const void*>(slab_h_batch_kernel<real, false>),
      reinterpret_cast<const void*>(slab_h_batch_kernel<real, true>),
  };
  for (const void* f : fns) {
    const cudaError_t err = cudaFuncGetAttributes(&fa, f);
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

#define OAFDTD_SLAB(real)                                                                                             \
  template int inject_blocks<real>(const EdgeArgs<real>&);                                                            \
  template cudaError_t preload_slab<real>();                                                                          \
  template cudaError_t slab_plan<real>(const SweepArgs<real>&, int, SlabLaunch*, long long*, int);                    \
  template long long slab_vecs<real>(const SweepArgs<real>&, int);                                                    \
  template bool slab_thin<real>(const SweepArgs<real>&, int);                                                         \
  template cudaError_t launch_slab_batch<real>(const SweepArgs<real>*, const SlabLaunch*, const EdgeArgs<real>*,      \
                                               const ProbeArgs<real>*, const BatchGrid&, int, int, bool, bool, int,   \
                                               bool, cudaStream_t);                                                   \
  template cudaError_t launch_slab<real>(const SweepArgs<real>&, int, cudaStream_t, const EdgeArgs<real>*,            \
                                         const ProbeArgs<real>*, int, bool);
OAFDTD_SLAB(float)
OAFDTD_SLAB(double)

}  // namespace oafdtd
