// Volume kernels: one RK stage of the elastic velocity-stress system on one
// block.  Pre-kernels fold the boundary/fault penalties and the PML damping
// into DF, the stencil kernel does the bulk per grid point, and correction
// kernels add the sources, the attenuation and the plastic map:
//
//   DF <- A*DF + L(F)                 (scale_rates + set_rates,
//                                      src/fields.f90:49-108,
//                                      src/JU_xJU_yJU_z6.f90:12-812, 16141-16449,
//                                      src/RHS_Interior.f90:133-274)
//   DF -= PML damping, DQ <- A*DQ+..  (src/RHS_Interior.f90:1782-2201)
//   DF -= tau0/h * boundary SAT       (src/RHS_Interior.f90:1516-1703,
//                                      src/BoundaryConditions.f90:777-918 or
//                                      src/BoundaryConditions3.f90:777-903)
//   DF -= tau0/h * fault SAT          (src/RHS_Interior.f90:1706-1779; the SAT
//                                      vector comes from the interface kernel)
//   F_out = F_in + B*dt*DF            (update_fields, src/fields.f90:111-171;
//                                      Kahan-compensated in FP32 mode)
//   plastic return map on the last stage (src/plastic.f90:11-217)
//
// Curvilinear blocks use the conservative flux form for the stress
// divergence, D_d(J*metric*sigma)/(rho*J), and metric(centre)*D_d(v) for the
// velocity gradient; the three per-direction fluxes of each momentum
// component are combined before differencing (D is linear), so each point
// differences 6 quantities per axis.  Cartesian blocks use the diagonal
// constant metric.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <utility>

#include "wql_internal.h"
#include "wql_stencil.cuh"

namespace wql {
namespace {

// Load the six differenced quantities at point q for axis d: velocities
// and the momentum fluxes through the d-faces.
template <typename T, bool CURV>
__device__ __forceinline__ void load6(const T* __restrict__ F, const T* __restrict__ coef,
                                      long long np, long long q, int d, T o[6]) {
  o[0] = F[q];
  o[1] = F[np + q];
  o[2] = F[2 * np + q];
  if (CURV) {
    const T a = coef[(d * 3 + 0) * np + q], b = coef[(d * 3 + 1) * np + q],
            c = coef[(d * 3 + 2) * np + q];
    const T sxx = F[3 * np + q], syy = F[4 * np + q], szz = F[5 * np + q];
    const T sxy = F[6 * np + q], sxz = F[7 * np + q], syz = F[8 * np + q];
    o[3] = a * sxx + b * sxy + c * sxz;
    o[4] = a * sxy + b * syy + c * syz;
    o[5] = a * sxz + b * syz + c * szz;
  } else {
    o[3] = F[sig(0, d) * np + q];
    o[4] = F[sig(1, d) * np + q];
    o[5] = F[sig(2, d) * np + q];
  }
}

// ---------------------------------------------------------------------------
// Rows of the difference operators for the per-point kernels.  The weights of
// the block's operator sit in shared memory (the closure rows of neighbouring
// lanes differ, which constant memory would serve one row at a time):
//   FD 0  SBP-6: [row 6][point 9]
//   FD 1  upwind order 6: [D+, D-][row 6][point 10]
//   FD 2  upwind order 5: [D+, D-][row 4][point 7]
//   FD 3..5  a table operator whose interior rows lie within -(FD-1)..FD (D+)
//         and -FD..FD-1 (D-): the whole table (UpG), then the interior rows on
//         that window, [interior, shell][D+, D-][2*FD]
template <int FD>
constexpr int kRowWords = FD == 0 ? 54 : (FD == 1 ? 120 : (FD == 2 ? 56 : kUgWords + 8 * FD));

// The narrowest window that holds a table operator's interior rows (orders 2
// to 4 and DRP 3: 3; order 7, DRP 4, 5 and 66: 4; the others 5).
inline int ug_window(const UpG& g) {
  for (int w = 3; w < 5; ++w)
    if (g.plo >= 1 - w && g.plo + g.pn - 1 <= w && g.mlo >= -w && g.mlo + g.mn - 1 <= w - 1) return w;
  return 5;
}

template <typename T, int FD>
__device__ __forceinline__ void load_rows(T* tab, const UpG& g) {
  const int nt = blockDim.x * blockDim.y;
  for (int e = threadIdx.x + blockDim.x * threadIdx.y; e < kRowWords<FD>; e += nt) {
    if constexpr (FD == 0) tab[e] = sbp_w<T>(e / 9, e % 9);
    else if constexpr (FD == 1) tab[e] = up_w<T>(e / 60, e / 10 % 6, e % 10);
    else if constexpr (FD == 2) tab[e] = upw<T, 2>(e / 28, e / 7 % 4, e % 7);
    else if (e < kUgWords) tab[e] = ((const T*)g.w)[e];
    else {
      const int x = e - kUgWords, k = x % (2 * FD), minus = x / (2 * FD) & 1, set = x / (4 * FD);
      const int idx = k - (minus ? FD + g.mlo : FD - 1 + g.plo);
      tab[e] = idx >= 0 && idx < (minus ? g.mn : g.pn) ? ((const T*)g.w)[(2 * set + minus) * kUgCol + idx] : T(0);
    }
  }
  __syncthreads();
}

// Calls vel(offset, weight) and flux(offset, weight) for the points of the
// rows of the velocity and the flux operator at 0-based index i of n along
// axis d (one operator for both in FD 0, D+ and D- else).  The interior rows of
// FD 0 call vel2(offset, weight) and flux2(offset, weight) for the weighted
// difference of the points at +offset and -offset: differenced first, FP32
// fields lose less (4.2e-7 against 4.5e-7 in the velocities after 60 steps of
// 2 x 99x97x97).  Interior rows and
// closure columns are unrolled so that their loads are in flight together.
// shell (FD 3..5): the point lies in the boundary shell, whose interior rows are
// the near-boundary routine's.
template <typename T, int FD, typename V, typename X, typename V2, typename X2>
__device__ __forceinline__ void visit_row(const T* tab, const UpG& g, bool shell, int i, int n, int d, V&& vel,
                                          X&& flux, V2&& vel2, X2&& flux2) {
  if constexpr (FD >= 3) {
    if (i >= g.R && i < n - g.R) {
      // a fixed window with zero weights outside the operator's own: with the
      // operator's run-time bounds tested per offset, every offset waited for
      // its own loads.  Only rows nearer to an end than the window (orders 2
      // and 3, whose closures are shorter) clamp its points to the axis.
      const T* wp = tab + kUgWords + (shell ? 4 * FD : 0);
      if (i >= FD && i < n - FD) {
#pragma unroll
        for (int k = 0; k < 2 * FD; ++k) {
          vel(k + 1 - FD, wp[k]);
          flux(k - FD, wp[2 * FD + k]);
        }
      } else {
#pragma unroll 2
        for (int k = 0; k < 2 * FD; ++k) {
          vel(min(max(k + 1 - FD, -i), n - 1 - i), wp[k]);
          flux(min(max(k - FD, -i), n - 1 - i), wp[2 * FD + k]);
        }
      }
    } else {
      // left row i reads points 0.., right row k = n-1-i points n-1-t
      const bool left = i < g.R;
      const int row = left ? i : n - 1 - i;
      const T* wp = tab + 4 * kUgCol + (left ? 0 : 2 * kUgRowBlock) + (d * kUgRows + row) * kUgCol;
#pragma unroll 4
      for (int t = 0; t < kUgCol; ++t) {
        const int off = min(max(left ? t - row : row - t, -i), n - 1 - i);
        vel(off, wp[t]);
        flux(off, wp[kUgRowBlock + t]);
      }
    }
  } else {
    const int kind = FD ? up_kind<FD ? FD : 1>(i, n) : sbp_kind(i, n);
    if (kind == 0 && FD) {
      constexpr int PHI = UpOp<FD ? FD : 1>::PHI;
#pragma unroll
      for (int o = -PHI; o <= PHI; ++o) {
        if (o >= -2) vel(o, up_cf<T, FD ? FD : 1>(o));
        if (o <= 2) flux(o, -up_cf<T, FD ? FD : 1>(-o));
      }
    } else if (kind == 0) {
      const T cs[3] = {T(kC1), T(kC2), T(kC3)};
#pragma unroll
      for (int s = 1; s <= 3; ++s) {
        vel2(s, cs[s - 1]);
        flux2(s, cs[s - 1]);
      }
    } else {
      // left row kind = -1-row reads points 0.., right row kind = 1+row the
      // mirrored points with negated weights (the upwind pair swaps its two
      // tables there)
      constexpr int NC = FD ? UpOp<FD ? FD : 1>::NCOL : 9, NR = FD ? UpOp<FD ? FD : 1>::R : 6;
      const bool left = kind < 0;
      const int row = left ? -kind - 1 : kind - 1;
      const T sgn = left ? T(1) : T(-1);
      const T* wv = tab + (FD && !left ? NR * NC : 0) + row * NC;
      const T* wf = FD ? tab + (left ? NR * NC : 0) + row * NC : wv;
#pragma unroll(FD == 1 ? 5 : (FD == 2 ? 7 : 3))
      for (int t = 0; t < NC; ++t) {
        const int off = left ? t - row : row - t;
        // zero weights too: a test per column would put its latency before
        // the column's loads
        vel(off, sgn * wv[t]);
        flux(off, sgn * wf[t]);
      }
    }
  }
}

// Whether point idx lies in the boundary shell of a table operator: outside
// [lo, n-1-hi] on some axis, with lo and hi the closure rows R, or npml on a
// PML side if larger (the interior limits of the interior routines,
// src/RHS_Interior.f90:40-125, 276-1512).
template <typename T>
__device__ __forceinline__ bool ug_shell(const VolumeArgs<T>& a, int i, int j, int k) {
  bool shell = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int idx = d == 0 ? i : (d == 1 ? j : k), n = d == 0 ? a.nq : (d == 1 ? a.nr : a.ns);
    const int lo = a.pml[2 * d] ? max(a.ug.R, a.npml) : a.ug.R;
    const int hi = a.pml[2 * d + 1] ? max(a.ug.R, a.npml) : a.ug.R;
    shell = shell || idx < lo || idx > n - 1 - hi;
  }
  return shell;
}

// Whether the pre-kernels have set DF of the point on a stage with A = 0: a
// block face or a PML slab.
template <typename T>
__device__ __forceinline__ bool df_set(const VolumeArgs<T>& a, int i, int j, int k) {
  const int w = a.npml;
  return i == 0 || i == a.nq - 1 || j == 0 || j == a.nr - 1 || k == 0 || k == a.ns - 1 || (a.pml[0] && i < w) ||
         (a.pml[1] && i >= a.nq - w) || (a.pml[2] && j < w) || (a.pml[3] && j >= a.nr - w) || (a.pml[4] && k < w) ||
         (a.pml[5] && k >= a.ns - w);
}

// Two blocks' arguments of a launch over one block or a scenario's two.
template <typename T>
struct BlockPair {
  VolumeArgs<T> a[2];
  long long n0;  // threads, planes or CTAs of block 0 (by the kernel)
};

// ---------------------------------------------------------------------------
// Main stencil kernel (2.5-D tiled).  Computes, for every point of the block,
//   DF <- A*DF + L(F)      and      F_out <- F + B*dt*DF
// (scale_rates + set_rates + update_fields, src/fields.f90:49-171,
// src/JU_xJU_yJU_z6.f90:12-812 and 16141-16449, src/RHS_Interior.f90:133-274),
// with the Kahan-compensated update in FP32C mode.  Boundary penalties and the
// PML damping are folded into DF beforehand by the pre-kernels below (they are
// linear in DF, so the order of the sums changes only rounding).
//
// A CTA of TQ x TR threads owns a (q,r) tile and marches along s through a
// chunk of planes.  Per plane the tile plus a 3-point halo in q and r is
// staged into shared memory as the differenced quantities -- velocities and
// the q- and r-face momentum fluxes J*metric*sigma -- so each is formed once
// and read by up to 7 neighbours from shared memory.  Along s every thread
// keeps (v, s-face flux) of a 9-plane window in private shared-memory slots,
// enough for the 7-point central rows and for the one-sided closure rows,
// which read planes 0..8 (or n-9..n-1).  The last tile along q and r is
// shifted to end on the last point and owns its whole width, so every
// closure row lies inside one tile plus halo (needs TQ, TR >= 8).
template <typename T, int TQ, int TR>
struct Tile {
  static constexpr int HQ = TQ + 6, HR = TR + 6, NRING = 9;
  static constexpr int sgq_off = 3 * HR * HQ, sgr_off = sgq_off + 3 * TR * HQ, ring_off = sgr_off + 3 * HR * TQ;
  static constexpr size_t words = ring_off + NRING * 6 * TR * TQ;
  __device__ static T& sv(T* b, int c, int lr, int lq) { return b[(c * HR + lr) * HQ + lq]; }
  __device__ static T& sgq(T* b, int c, int ty, int lq) { return b[sgq_off + (c * TR + ty) * HQ + lq]; }
  __device__ static T& sgr(T* b, int c, int lr, int tx) { return b[sgr_off + (c * HR + lr) * TQ + tx]; }
  __device__ static T& ring(T* b, int slot, int c, int ty, int tx) {
    return b[ring_off + ((slot * 6 + c) * TR + ty) * TQ + tx];
  }
};

template <typename T, bool CURV, bool KAHAN, int TQ, int TR, int MINB>
__global__ void __launch_bounds__(TQ * TR, MINB) stencil_kernel_tiled(const __grid_constant__ VolumeArgs<T> a,
                                                                       int schunk) {
  using TL = Tile<T, TQ, TR>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int nq = a.nq, nr = a.nr, ns = a.ns;
  const long long np = a.np;
  const long long sts = (long long)a.pq * nr;
  const TileSpan spq = tile_span(blockIdx.x, nq, TQ), spr = tile_span(blockIdx.y, nr, TR);
  const int q0 = spq.origin, r0 = spr.origin;
  const int q = q0 + tx, r = r0 + ty;
  const bool valid = q < nq && r < nr;
  const bool own = valid && q >= spq.own_lo && q < spq.own_hi && r >= spr.own_lo && r < spr.own_hi;
  const int s_begin = blockIdx.z * schunk;
  const int s_end = min(ns, s_begin + schunk);
  const T* __restrict__ F = a.Fin;
  const T* __restrict__ coef = a.coef;
  const int lq = tx + 3, lr = ty + 3;
  const int kq = sbp_kind(q, nq), kr = sbp_kind(r, nr);
  const long long col = q + (long long)a.pq * r;
  int lo = 0, hi = -1;  // planes held by the ring (uniform across the CTA)

  for (int s = s_begin; s < s_end; ++s) {
    const long long p = col + sts * s;
    // ---- ring: make planes [need_lo, need_hi] resident (private slots)
    const int ks = sbp_kind(s, ns);
    const int need_lo = ks < 0 ? 0 : (ks > 0 ? ns - 9 : s - 3);
    const int need_hi = ks < 0 ? 8 : (ks > 0 ? ns - 1 : s + 3);
    if (need_lo < lo || need_lo > hi + 1) {
      lo = need_lo;
      hi = need_lo - 1;
    }
    for (int pl = hi + 1; pl <= need_hi; ++pl) {
      if (valid) {
        T t6[6];
        load6<T, CURV>(F, coef, np, col + sts * pl, 2, t6);
        const int slot = pl % 9;
#pragma unroll
        for (int c = 0; c < 6; ++c) TL::ring(sm, slot, c, ty, tx) = t6[c];
      }
    }
    hi = need_hi;
    lo = max(lo, hi - 8);
    // ---- stage the plane's cross region into shared memory
    __syncthreads();
    auto stage = [&](int gq, int gr, int lq_, int lr_, bool wq, bool wr) {
      const long long pp = gq + (long long)a.pq * gr + sts * s;
      T f[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) f[c] = F[c * np + pp];
#pragma unroll
      for (int c = 0; c < 3; ++c) TL::sv(sm, c, lr_, lq_) = f[c];
      if (wq) {
        if (CURV) {
          const T a0 = coef[0 * np + pp], a1 = coef[1 * np + pp], a2 = coef[2 * np + pp];
#pragma unroll
          for (int c = 0; c < 3; ++c)
            TL::sgq(sm, c, lr_ - 3, lq_) = a0 * f[sig(c, 0)] + a1 * f[sig(c, 1)] + a2 * f[sig(c, 2)];
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) TL::sgq(sm, c, lr_ - 3, lq_) = f[sig(c, 0)];
        }
      }
      if (wr) {
        if (CURV) {
          const T a0 = coef[3 * np + pp], a1 = coef[4 * np + pp], a2 = coef[5 * np + pp];
#pragma unroll
          for (int c = 0; c < 3; ++c)
            TL::sgr(sm, c, lr_, lq_ - 3) = a0 * f[sig(c, 0)] + a1 * f[sig(c, 1)] + a2 * f[sig(c, 2)];
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) TL::sgr(sm, c, lr_, lq_ - 3) = f[sig(c, 1)];
        }
      }
    };
    if (valid) stage(q, r, lq, lr, true, true);
    if (r < nr) {
      if (tx < 3 && q0 - 3 + tx >= 0) stage(q0 - 3 + tx, r, tx, lr, true, false);
      if (tx >= TQ - 3 && q0 + TQ + (tx - (TQ - 3)) < nq)
        stage(q0 + TQ + (tx - (TQ - 3)), r, TQ + 3 + (tx - (TQ - 3)), lr, true, false);
    }
    if (q < nq) {
      if (ty < 3 && r0 - 3 + ty >= 0) stage(q, r0 - 3 + ty, lq, ty, false, true);
      if (ty >= TR - 3 && r0 + TR + (ty - (TR - 3)) < nr)
        stage(q, r0 + TR + (ty - (TR - 3)), lq, TR + 3 + (ty - (TR - 3)), false, true);
    }
    __syncthreads();
    if (!own) continue;

    // ---- derivatives, consumed axis by axis
    T g[3][3], dv[3];
    const T Jinv = CURV ? coef[9 * np + p] : T(1);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      T o[6];
      const int kind = d == 0 ? kq : (d == 1 ? kr : ks);
      if (kind == 0) {
        const T c1 = T(kC1), c2 = T(kC2), c3 = T(kC3);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          T xp1, xm1, xp2, xm2, xp3, xm3;
          if (d == 0) {
            auto X = [&](int l) -> T { return c < 3 ? TL::sv(sm, c, lr, l) : TL::sgq(sm, c - 3, ty, l); };
            xp1 = X(lq + 1); xm1 = X(lq - 1); xp2 = X(lq + 2); xm2 = X(lq - 2); xp3 = X(lq + 3); xm3 = X(lq - 3);
          } else if (d == 1) {
            auto X = [&](int l) -> T { return c < 3 ? TL::sv(sm, c, l, lq) : TL::sgr(sm, c - 3, l, tx); };
            xp1 = X(lr + 1); xm1 = X(lr - 1); xp2 = X(lr + 2); xm2 = X(lr - 2); xp3 = X(lr + 3); xm3 = X(lr - 3);
          } else {
            xp1 = TL::ring(sm, (s + 1) % 9, c, ty, tx); xm1 = TL::ring(sm, (s + 8) % 9, c, ty, tx);
            xp2 = TL::ring(sm, (s + 2) % 9, c, ty, tx); xm2 = TL::ring(sm, (s + 7) % 9, c, ty, tx);
            xp3 = TL::ring(sm, (s + 3) % 9, c, ty, tx); xm3 = TL::ring(sm, (s + 6) % 9, c, ty, tx);
          }
          o[c] = c1 * (xp1 - xm1) + c2 * (xp2 - xm2) + c3 * (xp3 - xm3);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 6; ++c) o[c] = T(0);
#pragma unroll 1
        for (int t = 0; t < 9; ++t) {
          T w;
          int off;
          row_entry<T>(kind, t, w, off);
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            T x;
            if (d == 0) x = c < 3 ? TL::sv(sm, c, lr, lq + off) : TL::sgq(sm, c - 3, ty, lq + off);
            else if (d == 1) x = c < 3 ? TL::sv(sm, c, lr + off, lq) : TL::sgr(sm, c - 3, lr + off, tx);
            else x = TL::ring(sm, (s + off + 18) % 9, c, ty, tx);
            o[c] += w * x;
          }
        }
      }
      const T rh = a.rh[d];
      if (CURV) {
        T m[3];
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) m[jj] = coef[(d * 3 + jj) * np + p] * Jinv;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          dv[c] = d == 0 ? rh * o[3 + c] : dv[c] + rh * o[3 + c];
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) g[c][jj] = d == 0 ? m[jj] * (rh * o[c]) : g[c][jj] + m[jj] * (rh * o[c]);
        }
      } else {
        const T sc = a.cart_metric[d] * rh;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          dv[c] = d == 0 ? sc * o[3 + c] : dv[c] + sc * o[3 + c];
          g[c][d] = sc * o[c];
        }
      }
    }
    T lam, mu, rinv;
    if (CURV) {
      lam = coef[10 * np + p];
      mu = coef[11 * np + p];
      rinv = coef[12 * np + p];
    } else {
      lam = coef[0 * np + p];
      mu = coef[1 * np + p];
      rinv = coef[2 * np + p];
    }
    const T l2m = lam + T(2) * mu;
    T du[9];
    du[0] = rinv * dv[0];
    du[1] = rinv * dv[1];
    du[2] = rinv * dv[2];
    du[3] = l2m * g[0][0] + lam * (g[1][1] + g[2][2]);
    du[4] = l2m * g[1][1] + lam * (g[0][0] + g[2][2]);
    du[5] = l2m * g[2][2] + lam * (g[0][0] + g[1][1]);
    du[6] = mu * (g[0][1] + g[1][0]);
    du[7] = mu * (g[0][2] + g[2][0]);
    du[8] = mu * (g[1][2] + g[2][1]);
    const bool keep = a.A != T(0), set = !keep && df_set(a, q, r, s);
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      const T f0 = F[c * np + p];
      const T df = (keep ? a.A * a.DF[c * np + p] : (set ? a.DF[c * np + p] : T(0))) + du[c];
      a.DF[c * np + p] = df;
      if (KAHAN) {
        const T y = a.Bdt * df - (T)comp_get(a.C, c * np + p);
        const T t = f0 + y;
        comp_put(a.C, c * np + p, (float)((t - f0) - y));
        a.Fout[c * np + p] = t;
      } else {
        a.Fout[c * np + p] = f0 + a.Bdt * df;
      }
    }
  }
}

// Per-point form of the same stencil kernel: every neighbour value is read
// through L1/L2.  It runs the upwind operators that the TMA kernel does not
// take (the table operators, order 5, and FP64) and serves as a cross-check
// of the other kernels.  One launch covers one block or a scenario's two:
// planes [0, n0) of the grid are block 0's.
template <typename T, bool CURV, bool KAHAN, int FD = 0>
__global__ void __launch_bounds__(256) stencil_kernel_pointwise(const __grid_constant__ BlockPair<T> P) {
  __shared__ T tab[kRowWords<FD>];
  load_rows<T, FD>(tab, P.a[0].ug);
  const int blk = (long long)blockIdx.z >= P.n0 ? 1 : 0;
  const VolumeArgs<T>& a = P.a[blk];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = (int)blockIdx.z - (blk ? (int)P.n0 : 0);
  if (i >= a.nq || j >= a.nr) return;
  const long long np = a.np;
  const long long p = i + (long long)a.pq * (j + (long long)a.nr * k);
  const T* __restrict__ F = a.Fin + p;
  const T* __restrict__ coef = a.coef + p;
  // neighbours: a component's uniform base and one 32-bit index that all of
  // the neighbour's components share
  const T* __restrict__ Fu = a.Fin;
  const T* __restrict__ Cu = a.coef;
  const unsigned pu = (unsigned)p;
  T g[3][3], dv[3];
  const T Jinv = CURV ? coef[9 * np] : T(1);
  const bool shell = FD >= 3 && ug_shell(a, i, j, k);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const unsigned st = d == 0 ? 1u : (d == 1 ? (unsigned)a.pq : (unsigned)a.pq * (unsigned)a.nr);
    T o[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) o[c] = T(0);
    visit_row<T, FD>(
        tab, a.ug, shell, d == 0 ? i : (d == 1 ? j : k), d == 0 ? a.nq : (d == 1 ? a.nr : a.ns), d,
        [&](int off, T w) {
          const unsigned q = pu + (unsigned)off * st;
#pragma unroll
          for (int c = 0; c < 3; ++c) o[c] += w * (Fu + c * np)[q];
        },
        [&](int off, T w) {
          const unsigned q = pu + (unsigned)off * st;
          if (CURV) {
            // the weight goes to the flux, not into its metrics (rounded there,
            // it is off by the same at every point of a regular grid)
            const T m0 = (Cu + (d * 3) * np)[q], m1 = (Cu + (d * 3 + 1) * np)[q], m2 = (Cu + (d * 3 + 2) * np)[q];
#pragma unroll
            for (int c = 0; c < 3; ++c)
              o[3 + c] += w * (m0 * (Fu + sig(c, 0) * np)[q] + m1 * (Fu + sig(c, 1) * np)[q] +
                               m2 * (Fu + sig(c, 2) * np)[q]);
          } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) o[3 + c] += w * (Fu + sig(c, d) * np)[q];
          }
        },
        [&](int off, T w) {
          const unsigned h = pu + (unsigned)off * st, l = pu - (unsigned)off * st;
#pragma unroll
          for (int c = 0; c < 3; ++c) o[c] += w * ((Fu + c * np)[h] - (Fu + c * np)[l]);
        },
        [&](int off, T w) {
          const unsigned h = pu + (unsigned)off * st, l = pu - (unsigned)off * st;
          T x[2][3];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const unsigned q = e ? l : h;
            T m[3] = {T(0), T(0), T(0)};
#pragma unroll
            for (int j = 0; CURV && j < 3; ++j) m[j] = (Cu + (d * 3 + j) * np)[q];
#pragma unroll
            for (int c = 0; c < 3; ++c)
              x[e][c] = CURV ? m[0] * (Fu + sig(c, 0) * np)[q] + m[1] * (Fu + sig(c, 1) * np)[q] +
                                   m[2] * (Fu + sig(c, 2) * np)[q]
                             : (Fu + sig(c, d) * np)[q];
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) o[3 + c] += w * (x[0][c] - x[1][c]);
        });
    const T rh = a.rh[d];
    if (CURV) {
      T m[3];
#pragma unroll
      for (int jj = 0; jj < 3; ++jj) m[jj] = coef[(d * 3 + jj) * np] * Jinv;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        dv[c] = d == 0 ? rh * o[3 + c] : dv[c] + rh * o[3 + c];
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) g[c][jj] = d == 0 ? m[jj] * (rh * o[c]) : g[c][jj] + m[jj] * (rh * o[c]);
      }
    } else {
      const T sc = a.cart_metric[d] * rh;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        dv[c] = d == 0 ? sc * o[3 + c] : dv[c] + sc * o[3 + c];
        g[c][d] = sc * o[c];
      }
    }
  }
  const T lam = coef[(CURV ? 10 : 0) * np];
  const T mu = coef[(CURV ? 11 : 1) * np];
  const T rinv = coef[(CURV ? 12 : 2) * np];
  const T l2m = lam + T(2) * mu;
  T du[9];
  du[0] = rinv * dv[0];
  du[1] = rinv * dv[1];
  du[2] = rinv * dv[2];
  du[3] = l2m * g[0][0] + lam * (g[1][1] + g[2][2]);
  du[4] = l2m * g[1][1] + lam * (g[0][0] + g[2][2]);
  du[5] = l2m * g[2][2] + lam * (g[0][0] + g[1][1]);
  du[6] = mu * (g[0][1] + g[1][0]);
  du[7] = mu * (g[0][2] + g[2][0]);
  du[8] = mu * (g[1][2] + g[2][1]);
  const bool keep = a.A != T(0), set = !keep && df_set(a, i, j, k);
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    const T f0 = F[c * np];
    const T df = (keep ? a.A * a.DF[c * np + p] : (set ? a.DF[c * np + p] : T(0))) + du[c];
    a.DF[c * np + p] = df;
    if (KAHAN) {
      const T y = a.Bdt * df - (T)comp_get(a.C, c * np + p);
      const T t = f0 + y;
      comp_put(a.C, c * np + p, (float)((t - f0) - y));
      a.Fout[c * np + p] = t;
    } else {
      a.Fout[c * np + p] = f0 + a.Bdt * df;
    }
  }
}

// Offset of block point (i, j, k) within the slab of `side`.
template <typename T>
__device__ __forceinline__ long long slab_point(const VolumeArgs<T>& a, int side, int i, int j, int k) {
  const int axis = side >> 1, npml = a.npml;
  const bool hi = side & 1;
  if (axis == 0) return (hi ? i - (a.nq - npml) : i) + (long long)npml * (j + (long long)a.nr * k);
  if (axis == 1) return i + (long long)a.nq * ((hi ? j - (a.nr - npml) : j) + (long long)npml * k);
  return i + (long long)a.nq * (j + (long long)a.nr * (hi ? k - (a.ns - npml) : k));
}

// ---------------------------------------------------------------------------
// PML pre-kernel (src/RHS_Interior.f90:1782-2201, src/fields.f90:70-105,
// 131-166): for every point inside one or more active slabs, the damping terms
// of the rates, DQ <- A*DQ + sources - (d+cfs)*Q and Q <- Q + B*dt*DQ.  It
// runs before the stencil of its stage.  Everything it needs is stage input
// (F, Q, DQ), so the damping terms are folded into DF (DF + corr/A, or corr
// on a stage with A = 0) and the stencil's A*DF + du carries them: F_out and
// its compensation are not read and written a second time, and no velocity
// gradient is handed over.  The face pre-kernel, which runs first, has folded
// the boundary forcing of the auxiliary fields into DQ at the slab's own face.
//
// The slab union is cut into regions along the slab edges, up to 26, so that
// the sides a point lies in are the same for a whole CTA: the axis of a side
// and the arrays of its fluxes are uniform, and every load of a neighbour is
// a uniform base plus one 32-bit offset that all of the neighbour's
// quantities share.  A CTA takes a tile of 256 points of one region, 4 to 32
// points along q and 2 to 8 along r and s, whichever pads the region least:
// neighbouring rows share their stencil reads in L1.  Each direction's
// neighbours are visited once for both the flux and the velocity derivative; a
// closure row's columns are unrolled like the interior row's, so their loads
// are in flight together (as a loop, their latencies added up).  At the 80
// registers of three CTAs an SM every FP32 form spills 80 to 370 bytes a thread
// (stores); with two CTAs and no spills the slabs take longer (2 x 401x201^2:
// 13.8 ms a step against 12.95).
struct PmlTiles {
  int n;
  int lo[26][3], dim[26][3];
  int sides[26];       // bit per side
  int lw[26], lr[26];  // log2 of the tile extents along q and r
  int tq[26], tr[26];  // tiles along q and r
  int start[27];       // CTAs before region b
};

template <typename T>
PmlTiles pml_tiles(const VolumeArgs<T>& a) {
  PmlTiles P;
  P.n = 0;
  P.start[0] = 0;
  const int nn[3] = {a.nq, a.nr, a.ns}, w = a.npml;
  // the intervals of each axis between its slab edges, with the sides they lie in
  int cut[3][4], m[3], in[3][3];
  for (int d = 0; d < 3; ++d) {
    int e[4] = {0, a.pml[2 * d] ? w : 0, a.pml[2 * d + 1] ? nn[d] - w : nn[d], nn[d]};
    if (e[1] > e[2]) std::swap(e[1], e[2]);
    m[d] = 0;
    cut[d][0] = 0;
    for (int k = 0; k < 3; ++k) {
      if (e[k + 1] <= e[k]) continue;
      in[d][m[d]] = (a.pml[2 * d] && e[k] < w ? 1 << (2 * d) : 0) |
                    (a.pml[2 * d + 1] && e[k] >= nn[d] - w ? 2 << (2 * d) : 0);
      cut[d][++m[d]] = e[k + 1];
    }
  }
  for (int z = 0; z < m[2]; ++z)
    for (int y = 0; y < m[1]; ++y)
      for (int x = 0; x < m[0]; ++x) {
        const int sides = in[0][x] | in[1][y] | in[2][z], b = P.n;
        if (!sides) continue;
        const int c[3] = {x, y, z};
        for (int d = 0; d < 3; ++d) {
          P.lo[b][d] = cut[d][c[d]];
          P.dim[b][d] = cut[d][c[d] + 1] - cut[d][c[d]];
        }
        P.sides[b] = sides;
        if (sizeof(T) == 8) {  // the FP64 unit is the bound: no idle lanes, 256 consecutive points
          const long long pts = (long long)P.dim[b][0] * P.dim[b][1] * P.dim[b][2];
          P.tq[b] = P.tr[b] = 1;
          P.lw[b] = P.lr[b] = 0;
          P.start[b + 1] = P.start[b] + (int)((pts + 255) / 256);
          ++P.n;
          continue;
        }
        // the tile of 256 points that pads the region least; rows of 4 points
        // half use their 32-byte sectors
        float least = 1e30f;
        int ls = 0;
        for (int w2 = 5; w2 >= 2; --w2)
          for (int r2 = 3; r2 >= 1; --r2) {
            const int s2 = 8 - w2 - r2;
            if (s2 < 1 || s2 > 3) continue;
            auto up = [](int n, int l) { return (float)(((n + (1 << l) - 1) >> l) << l); };
            const float v = up(P.dim[b][0], w2) * up(P.dim[b][1], r2) * up(P.dim[b][2], s2) * (w2 == 2 ? 1.1f : 1.0f);
            if (v < 0.999f * least) {
              least = v;
              P.lw[b] = w2;
              P.lr[b] = r2;
              ls = s2;
            }
          }
        P.tq[b] = (P.dim[b][0] + (1 << P.lw[b]) - 1) >> P.lw[b];
        P.tr[b] = (P.dim[b][1] + (1 << P.lr[b]) - 1) >> P.lr[b];
        const int ts = (P.dim[b][2] + (1 << ls) - 1) >> ls;
        P.start[b + 1] = P.start[b] + P.tq[b] * P.tr[b] * ts;
        ++P.n;
      }
  return P;
}

// One or two blocks in a launch: CTAs [0, n0) take block 0's tiles.
template <typename T>
struct PmlPair {
  VolumeArgs<T> a[2];
  PmlTiles t[2];
  int n0;
};

// Element at a byte offset; O is unsigned, or size_t where a component is 4
// GiB or more (and for FP64 fields, whose kernel waits on the FP64 unit, not
// on address arithmetic).
template <typename T, typename O>
__device__ __forceinline__ T& at(T* base, O byte) {
  return *reinterpret_cast<T*>(reinterpret_cast<char*>(base) + byte);
}
template <typename T, typename O>
__device__ __forceinline__ T at(const T* base, O byte) {
  return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + byte);
}

template <typename T, typename O, bool CURV, int FD>
__device__ __forceinline__ void pml_pre_point(const VolumeArgs<T>& a, int i, int j, int k, unsigned sides,
                                              const T* tab) {
  const int nq = a.nq, nr = a.nr, ns = a.ns, npml = a.npml;
  const long long np = a.np;
  const O o = (O)sizeof(T) * ((O)i + (O)a.pq * ((O)j + (O)nr * (O)k));  // byte offset of the point in a component
  const T* __restrict__ F = a.Fin;
  const T* __restrict__ coef = a.coef;
  const T Jinv = CURV ? at(coef + 9 * np, o) : T(1);
  const T lam = at(coef + (CURV ? 10 : 0) * np, o), mu = at(coef + (CURV ? 11 : 1) * np, o);
  const T rinv = at(coef + (CURV ? 12 : 2) * np, o);
  const T rhoinv = CURV ? rinv / Jinv : rinv;
  const bool shell = FD >= 3 && ug_shell(a, i, j, k);
  // on a stage with A = 0, DF and DQ hold only what the face pre-kernel put there
  const bool keep = a.A != T(0);
  T corr[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) corr[c] = T(0);
  // one side; the axis is a compile-time constant so that the bases of all
  // loads are uniform
  auto take_side = [&](auto ax, const bool hi) {
    constexpr int axis = decltype(ax)::value;
    const int side = 2 * axis + (hi ? 1 : 0);
    const int ii = axis == 0 ? i : (axis == 1 ? j : k), n = axis == 0 ? nq : (axis == 1 ? nr : ns);
    // flux components of physical axis `axis`: sigma_{c,axis}
    const T* __restrict__ S0 = F + (axis == 0 ? 3 : (axis == 1 ? 6 : 7)) * np;
    const T* __restrict__ S1 = F + (axis == 0 ? 6 : (axis == 1 ? 4 : 8)) * np;
    const T* __restrict__ S2 = F + (axis == 0 ? 7 : (axis == 1 ? 8 : 5)) * np;
    T sd[3] = {T(0), T(0), T(0)}, gv[3] = {T(0), T(0), T(0)};
    // derivative along computational axis d of the velocities (o6[0..2]) and
    // of the fluxes J*metric_axis(d)*sigma_{c,axis} (o6[3..5])
    auto direction = [&](int d) {
      const O st = (O)sizeof(T) * (d == 0 ? (O)1 : (d == 1 ? (O)a.pq : (O)a.pq * (O)nr));
      const T* __restrict__ M = CURV ? coef + (d * 3 + axis) * np : coef;
      T o6[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) o6[c] = T(0);
      visit_row<T, FD>(
          tab, a.ug, shell, d == 0 ? i : (d == 1 ? j : k), d == 0 ? nq : (d == 1 ? nr : ns), d,
          [&](int off, T w) {
            const O q = o + (O)off * st;
#pragma unroll
            for (int c = 0; c < 3; ++c) o6[c] += w * at(F + c * np, q);
          },
          [&](int off, T w) {
            const O q = o + (O)off * st;
            const T m = CURV ? w * at(M, q) : w;
            o6[3] += m * at(S0, q);
            o6[4] += m * at(S1, q);
            o6[5] += m * at(S2, q);
          },
          [&](int off, T w) {
            const O h = o + (O)off * st, l = o - (O)off * st;
#pragma unroll
            for (int c = 0; c < 3; ++c) o6[c] += w * (at(F + c * np, h) - at(F + c * np, l));
          },
          [&](int off, T w) {
            const O h = o + (O)off * st, l = o - (O)off * st;
            const T mh = CURV ? at(M, h) : T(1), ml = CURV ? at(M, l) : T(1);
            o6[3] += w * (mh * at(S0, h) - ml * at(S0, l));
            o6[4] += w * (mh * at(S1, h) - ml * at(S1, l));
            o6[5] += w * (mh * at(S2, h) - ml * at(S2, l));
          });
      const T rh = a.rh[d];
      const T mt = rh * (CURV ? at(M, o) * Jinv : a.cart_metric[d]);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        gv[c] += mt * o6[c];
        sd[c] += rh * o6[3 + c];
      }
    };
    if (CURV) {
#pragma unroll 1
      for (int d = 0; d < 3; ++d) direction(d);
    } else {
      direction(axis);
    }
    // Q and DQ are read after the derivatives (held across them, they spill)
    T qv[9], dq[9];
    const bool forced = (hi ? ii == n - 1 : ii == 0) && a.bc[side] >= 1 && a.bc[side] <= 3;
    const long long sp = slab_point(a, side, i, j, k), snp = hi ? a.slab_np[2 * axis + 1] : a.slab_np[2 * axis];
    T* __restrict__ Q = (hi ? a.Q[2 * axis + 1] : a.Q[2 * axis]) + sp;
    T* __restrict__ DQ = (hi ? a.DQ[2 * axis + 1] : a.DQ[2 * axis]) + sp;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      qv[c] = Q[c * snp];
      dq[c] = keep || forced ? DQ[c * snp] : T(0);
    }
    const T sc = CURV ? Jinv : a.cart_metric[axis];
    // damping profile in grid-index units (src/RHS_Interior.f90:1855,1973,2092)
    const int off = hi ? ii + 1 - (n - npml) : (axis == 2 ? ii + 1 - npml : ii - npml);
    const T damp = a.pml_dn * (T)abs(off);
    const T cfs = T(1);
    const T dr = damp * rhoinv, dm = mu * damp;
    const T tr = damp * (lam * (qv[3] + qv[4] + qv[5])), d2 = dm + dm;
    corr[0] -= dr * qv[0];
    corr[1] -= dr * qv[1];
    corr[2] -= dr * qv[2];
    corr[3] -= tr + d2 * qv[3];
    corr[4] -= tr + d2 * qv[4];
    corr[5] -= tr + d2 * qv[5];
    corr[6] -= dm * qv[6];
    corr[7] -= dm * qv[7];
    corr[8] -= dm * qv[8];
    // velocity-gradient sources (src/RHS_Interior.f90:1890-1907, 2008-2025, 2125-2142)
    T src[9];
    src[0] = sd[0] * sc;
    src[1] = sd[1] * sc;
    src[2] = sd[2] * sc;
    src[3] = axis == 0 ? gv[0] : T(0);
    src[4] = axis == 1 ? gv[1] : T(0);
    src[5] = axis == 2 ? gv[2] : T(0);
    src[6] = axis == 0 ? gv[1] : (axis == 1 ? gv[0] : T(0));
    src[7] = axis == 0 ? gv[2] : (axis == 2 ? gv[0] : T(0));
    src[8] = axis == 1 ? gv[2] : (axis == 2 ? gv[1] : T(0));
    const T dc = damp + cfs, Ak = keep ? a.A : T(1);
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      const T nw = Ak * dq[c] + (src[c] - dc * qv[c]);
      DQ[c * snp] = nw;
      Q[c * snp] = qv[c] + a.Bdt * nw;
    }
  };
#pragma unroll 1
  for (unsigned m = sides & 3; m; m &= m - 1) take_side(std::integral_constant<int, 0>{}, m & 1 ? false : true);
#pragma unroll 1
  for (unsigned m = sides >> 2 & 3; m; m &= m - 1) take_side(std::integral_constant<int, 1>{}, m & 1 ? false : true);
#pragma unroll 1
  for (unsigned m = sides >> 4 & 3; m; m &= m - 1) take_side(std::integral_constant<int, 2>{}, m & 1 ? false : true);
  const bool face = i == 0 || i == nq - 1 || j == 0 || j == nr - 1 || k == 0 || k == ns - 1;
  const T inv = a.Ainv;
  T df[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) df[c] = keep || face ? at(a.DF + c * np, o) : T(0);
#pragma unroll
  for (int c = 0; c < 9; ++c) at(a.DF + c * np, o) = df[c] + corr[c] * inv;
}

template <typename T, typename O, bool CURV, int FD>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) pml_pre_kernel(const __grid_constant__ PmlPair<T> P) {
  __shared__ T tab[kRowWords<FD>];
  load_rows<T, FD>(tab, P.a[0].ug);
  const int blk = (int)blockIdx.x >= P.n0 ? 1 : 0;
  const int t = (int)blockIdx.x - (blk ? P.n0 : 0);
  const PmlTiles& B = P.t[blk];
  int b = 0;
  while (b < B.n - 1 && t >= B.start[b + 1]) ++b;
  const int l = t - B.start[b], lw = B.lw[b], lr = B.lr[b];
  const int bq = l % B.tq[b], br = (l / B.tq[b]) % B.tr[b], bs = l / (B.tq[b] * B.tr[b]);
  const int e = threadIdx.x;
  int i = (bq << lw) + (e & ((1 << lw) - 1));
  int j = (br << lr) + ((e >> lw) & ((1 << lr) - 1));
  int k = (bs << (8 - lw - lr)) + (e >> (lw + lr));
  if (sizeof(T) == 8) {
    const int x = l * 256 + e;
    i = x % B.dim[b][0];
    j = x / B.dim[b][0] % B.dim[b][1];
    k = x / (B.dim[b][0] * B.dim[b][1]);
  }
  if (i >= B.dim[b][0] || j >= B.dim[b][1] || k >= B.dim[b][2]) return;
  pml_pre_point<T, O, CURV, FD>(P.a[blk], B.lo[b][0] + i, B.lo[b][1] + j, B.lo[b][2] + k, (unsigned)B.sides[b], tab);
}

template <typename T, typename O, bool CURV>
void launch_pml_pre_fd(const PmlPair<T>& P, unsigned g, cudaStream_t s) {
  switch (P.a[0].fd) {
    case 0: pml_pre_kernel<T, O, CURV, 0><<<g, 256, 0, s>>>(P); return;
    case 1: pml_pre_kernel<T, O, CURV, 1><<<g, 256, 0, s>>>(P); return;
    case 2: pml_pre_kernel<T, O, CURV, 2><<<g, 256, 0, s>>>(P); return;
    default: pml_pre_kernel<T, O, CURV, 5><<<g, 256, 0, s>>>(P); return;
  }
}

// Launches the PML pre-kernel over one block (a1 null) or two.
template <typename T>
int launch_pml_pre(const VolumeArgs<T>& a0, const VolumeArgs<T>* a1, bool curv, cudaStream_t s) {
  if (a0.npml == 0 && !(a1 && a1->npml)) return 0;
  PmlPair<T> P;
  const VolumeArgs<T>* a[2] = {&a0, a1 ? a1 : &a0};
  int n[2];
  bool wide = sizeof(T) == 8;
  for (int b = 0; b < 2; ++b) {
    P.a[b] = *a[b];
    P.t[b] = pml_tiles(*a[b]);
    n[b] = a[b]->npml > 0 ? P.t[b].start[P.t[b].n] : 0;
    wide = wide || a[b]->np >= (1LL << 30);
  }
  if (!a1) n[1] = 0;
  P.n0 = n[0];
  if (n[0] + n[1] == 0) return 0;
  const unsigned g = (unsigned)(n[0] + n[1]);
  if (wide) curv ? launch_pml_pre_fd<T, size_t, true>(P, g, s) : launch_pml_pre_fd<T, size_t, false>(P, g, s);
  else if constexpr (sizeof(T) == 4)
    curv ? launch_pml_pre_fd<T, unsigned, true>(P, g, s) : launch_pml_pre_fd<T, unsigned, false>(P, g, s);
  return 1;
}

// ---------------------------------------------------------------------------
// three CTAs per SM: 80 registers, no spills in FP32 (four would cap it at 64
// and spill; the FP64 forms spill 80 to 88 bytes at 80)
#ifndef WQL_ANEL_MINB
#define WQL_ANEL_MINB 3
#endif
// Anelastic kernel (response = 'anelastic'; src/RHS_Interior.f90:2390-2509,
// the interior terms of src/JU_xJU_yJU_z6.f90:16316-16346, src/fields.f90:
// 61-68 and 122-129), one thread per point: the stress rates lose the sum
// of the point's four memory variables, each memory variable's rate is
//   Deta <- A*Deta + (relaxed strain-rate forcing - eta) / tau
// and eta <- eta + B*dt*Deta.  Inside a PML slab the strain rates lose the
// damped auxiliary fields (pml_damping_and_q, src/RHS_Interior.f90:
// 2287-2387) of the stage's input.  The
// velocity gradient is formed here with the block's operator (blocks whose
// stencil hands it over take anelastic_comp_kernel).
template <typename T, bool CURV, bool KAHAN, int FD>
__global__ void __launch_bounds__(256, WQL_ANEL_MINB) anelastic_kernel(const __grid_constant__ VolumeArgs<T> a) {
  __shared__ T tab[kRowWords<FD>];
  load_rows<T, FD>(tab, a.ug);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  const int nq = a.nq, nr = a.nr, ns = a.ns, npml = a.npml;
  if (i >= nq || j >= nr) return;
  const long long np = a.np;
  const long long p = i + (long long)a.pq * (j + (long long)nr * k);
  const int idx[3] = {i, j, k}, nn[3] = {nq, nr, ns};
  const T* __restrict__ F = a.Fin;
  const T* __restrict__ coef = a.coef;
  const T Jinv = CURV ? coef[9 * np + p] : T(1);
  T g[3][3];
  {
    const bool shell = FD >= 3 && ug_shell(a, i, j, k);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const long long st = d == 0 ? 1 : (d == 1 ? (long long)a.pq : (long long)a.pq * nr);
      T o[3] = {T(0), T(0), T(0)};
      visit_row<T, FD>(
          tab, a.ug, shell, idx[d], nn[d], d,
          [&](int off, T w) {
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c] += w * F[c * np + p + off * st];
          },
          [](int, T) {},
          [&](int off, T w) {
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c] += w * (F[c * np + p + off * st] - F[c * np + p - off * st]);
          },
          [](int, T) {});
      const T rh = a.rh[d];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (CURV) {
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) {
            const T m = coef[(d * 3 + jj) * np + p] * Jinv;
            g[c][jj] = d == 0 ? m * (rh * o[c]) : g[c][jj] + m * (rh * o[c]);
          }
        } else {
          g[c][d] = a.cart_metric[d] * rh * o[c];
        }
      }
    }
  }
  // strain rates: exx, eyy, ezz, gxy, gxz, gyz and the trace
  T e[6];
  e[0] = g[0][0];
  e[1] = g[1][1];
  e[2] = g[2][2];
  e[3] = g[0][1] + g[1][0];
  e[4] = g[0][2] + g[2][0];
  e[5] = g[1][2] + g[2][1];
  bool in_pml = false;
#pragma unroll
  for (int side = 0; side < 6; ++side) {
    const int ax = side >> 1;
    if (a.pml[side] && ((side & 1) ? idx[ax] >= nn[ax] - npml : idx[ax] < npml)) in_pml = true;
  }
  if (in_pml) {
    // d * Q terms per axis (damping profile and slab indexing as the PML kernel)
    T dq[3][3] = {{T(0), T(0), T(0)}, {T(0), T(0), T(0)}, {T(0), T(0), T(0)}};
#pragma unroll
    for (int side = 0; side < 6; ++side) {
      if (!a.pml[side]) continue;
      const int axis = side >> 1;
      const bool hi = side & 1;
      const int ii = idx[axis], n = nn[axis];
      if (!(hi ? (ii >= n - npml) : (ii < npml))) continue;
      const int off = hi ? ii + 1 - (n - npml) : (axis == 2 ? ii + 1 - npml : ii - npml);
      const T damp = (T)a.pml_d0 * (fabs((T)off / (T)npml));
      const long long sp = slab_point(a, side, i, j, k);
      const long long snp = a.slab_np[side];
      const T* Q = a.Q[side];
      const T* DQ = a.DQ[side];
      // the stage-input Q: the PML pre-kernel has advanced it by B*dt*DQ,
      // which is taken back (to the rounding of Q)
      auto q_in = [&](int c) { return Q[c * snp + sp] - a.Bdt * DQ[c * snp + sp]; };
      // Q components of the normal strain and the two shear strains of this axis
      const int cn = 3 + axis;
      const int c1 = axis == 0 ? 6 : (axis == 1 ? 6 : 7);
      const int c2 = axis == 0 ? 7 : 8;
      dq[axis][0] = damp * q_in(cn);
      dq[axis][1] = damp * q_in(c1);
      dq[axis][2] = damp * q_in(c2);
    }
    e[0] = e[0] - dq[0][0];
    e[1] = e[1] - dq[1][0];
    e[2] = e[2] - dq[2][0];
    e[3] = e[3] - dq[0][1] - dq[1][1];  // gxy: Qx(7), Qy(7)
    e[4] = e[4] - dq[0][2] - dq[2][1];  // gxz: Qx(8), Qz(8)
    e[5] = e[5] - dq[1][2] - dq[2][2];  // gyz: Qy(9), Qz(9)
  }
  const T tr = e[0] + e[1] + e[2];
  const T lam = CURV ? coef[10 * np + p] : coef[0 * np + p];
  const T mu = CURV ? coef[11 * np + p] : coef[1 * np + p];
  const T qs = a.qsinv[p];
  const T qp = T(0.5) * qs;
  T corr[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) corr[c] = T(0);
  // the memory-variable streams do not overlap (restrict): a component's
  // loads need not wait for the previous component's stores
  T* __restrict__ eta = a.eta;
  T* __restrict__ deta = a.Deta;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    T ev[1][4], dv[1][4];  // this component's four mechanisms
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      ev[0][m] = eta[(c * 4 + m) * np + p];
      dv[0][m] = deta[(c * 4 + m) * np + p];
    }
    corr[3 + c] = -(ev[0][0] + ev[0][1] + ev[0][2] + ev[0][3]);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const T w = (T)a.an_w[m];
      const T force = c < 3 ? (w * T(2) * mu * qs) * e[c] + (w * ((lam + T(2) * mu) * qp - T(2) * mu * qs)) * tr
                            : w * mu * qs * e[c];
      const long long q = (c * 4 + m) * np + p;
      const T de = a.A * dv[0][m] + (force - ev[0][m]) / (T)a.an_tau[m];
      deta[q] = de;
      eta[q] = ev[0][m] + a.Bdt * de;
    }
  }
  add_correction<T, KAHAN>(a, p, corr);
}

// The same with the velocity gradient at hand (a.G): six threads a point, one
// per stress component, 64 consecutive points of the pitched block a CTA.  One
// thread a point walked the six components with 80
// registers and 24 warps an SM, each waiting on its 66 streams (0.204 ms a
// block of 76x101x151, 46 % of HBM); a component's loads are now all in flight
// in 48 warps, the index takes 32-bit divisions and an axis looks up one slab
// side (0.131 ms, 72 % of HBM in its 552 B a point; 0.174 with 64-bit
// divisions, 0.151 with a loop over the six sides, which spilled).
template <typename T, bool CURV, bool KAHAN>
__global__ void __launch_bounds__(384, 4) anelastic_comp_kernel(const __grid_constant__ VolumeArgs<T> a) {
  const long long p = (long long)blockIdx.x * 64 + (threadIdx.x & 63);
  const int c = threadIdx.x >> 6;  // stress component 3 + c
  const long long np = a.np;
  if (p >= np) return;
  // 32-bit divisions (a block has fewer than 2^32 points)
  const unsigned pu = (unsigned)p, jk = pu / (unsigned)a.pq;
  const int i = (int)(pu - jk * (unsigned)a.pq), k = (int)(jk / (unsigned)a.nr), j = (int)(jk - (unsigned)k * (unsigned)a.nr);
  if (i >= a.nq) return;
  const T* __restrict__ coef = a.coef + p;
  const T* __restrict__ G = a.G + p;
  T* __restrict__ eta = a.eta + 4 * c * np + p;
  T* __restrict__ deta = a.Deta + 4 * c * np + p;
  T ev[4], dv[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    ev[m] = eta[m * np];
    dv[m] = deta[m * np];
  }
  const T mu = coef[(CURV ? 11 : 1) * np], qs = a.qsinv[p];
  // the component's strain rate e (twice the shear strain) and the trace
  T e, tr = T(0), lam = T(0);
  if (c < 3) {
    const T g0 = G[0], g1 = G[4 * np], g2_ = G[8 * np];
    e = c == 0 ? g0 : (c == 1 ? g1 : g2_);
    tr = g0 + g1 + g2_;
    lam = coef[(CURV ? 10 : 0) * np];
  } else {
    e = c == 3 ? G[np] + G[3 * np] : (c == 4 ? G[2 * np] + G[6 * np] : G[5 * np] + G[7 * np]);
  }
#pragma unroll
  for (int axis = 0; axis < 3; ++axis) {
    const int ii = axis == 0 ? i : (axis == 1 ? j : k), n = axis == 0 ? a.nq : (axis == 1 ? a.nr : a.ns);
    // where the two slabs of an axis overlap, the + side's Q alone counts
    // (pml_damping_and_q takes the sides in turn, src/RHS_Interior.f90:2287-2387)
    const bool hi = a.pml[2 * axis + 1] && ii >= n - a.npml;
    if (!hi && !(a.pml[2 * axis] && ii < a.npml)) continue;
    // the axes of a shear component: xy 0 1, xz 0 2, yz 1 2
    if (c >= 3 && (c == 3 ? axis == 2 : (c == 4 ? axis == 1 : axis == 0))) continue;
    const int off = hi ? ii + 1 - (n - a.npml) : (axis == 2 ? ii + 1 - a.npml : ii - a.npml);
    const T damp = a.pml_dn * (T)abs(off);
    const long long snp = hi ? a.slab_np[2 * axis + 1] : a.slab_np[2 * axis];
    const long long q = (c < 3 ? 3 + axis : 3 + c) * snp + slab_point(a, 2 * axis + (hi ? 1 : 0), i, j, k);
    // the stage-input Q (see anelastic_kernel)
    const T dq = damp * ((hi ? a.Q[2 * axis + 1] : a.Q[2 * axis])[q] - a.Bdt * (hi ? a.DQ[2 * axis + 1] : a.DQ[2 * axis])[q]);
    if (c < 3) tr -= dq;
    if (c >= 3 || c == axis) e -= dq;
  }
  // (w 2 mu qs) e + w ((lam + 2 mu) qp - 2 mu qs) tr, or (w mu qs) e
  const T ms = mu * qs;
  const T f = c < 3 ? T(2) * ms * e + ((lam + T(2) * mu) * (T(0.5) * qs) - T(2) * ms) * tr : ms * e;
  const T corr = -(ev[0] + ev[1] + ev[2] + ev[3]);
  const long long o = (3 + c) * np + p;
  const T df = a.DF[o], f0 = a.Fout[o];
  const T ck = KAHAN ? (T)comp_get(a.C, o) : T(0);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const T de = a.A * dv[m] + ((T)a.an_w[m] * f - ev[m]) * a.an_tinv[m];
    deta[m * np] = de;
    eta[m * np] = ev[m] + a.Bdt * de;
  }
  a.DF[o] = df + corr;
  if (KAHAN) {
    const T y = a.Bdt * corr - ck, t = f0 + y;
    comp_put(a.C, o, (float)((t - f0) - y));
    a.Fout[o] = t;
  } else {
    a.Fout[o] = f0 + a.Bdt * corr;
  }
}

// ---------------------------------------------------------------------------
// With a manufactured solution the boundary penalty acts on the fields less
// the exact solution at the stage's time (u = F - switch*fu,
// src/BoundaryConditions.f90:86-92, 126).
template <typename T>
__device__ __forceinline__ void mms_deviation(const VolumeArgs<T>& a, long long p, T (&u)[9]) {
  if (!a.ms) return;
  const T sv = a.mms_T * a.ms[p], ss = a.mms_T * a.ms[a.np + p];
#pragma unroll
  for (int c = 0; c < 9; ++c) u[c] -= c < 3 ? sv : ss;
}

// Manufactured-solution forcing (mms_forcing, src/mms.f90:77-133, which the
// reference never calls): DF -= T(t) mp - T'(t) S at every point of the
// block, with the matching update of F_out.
template <typename T, bool KAHAN>
__global__ void __launch_bounds__(256) mms_kernel(const __grid_constant__ VolumeArgs<T> a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (i >= a.nq || j >= a.nr) return;
  const long long np = a.np;
  const long long p = i + (long long)a.pq * (j + (long long)a.nr * k);
  const T sv = a.ms[p], ss = a.ms[np + p];
  T corr[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) corr[c] = -(a.mms_T * a.mp[c * np + p] - a.mms_Tp * (c < 3 ? sv : ss));
  add_correction<T, KAHAN>(a, p, corr);
}

// ---------------------------------------------------------------------------
// Face pre-kernel: the outer-boundary SAT (src/RHS_Interior.f90:1516-1703 with
// src/BoundaryConditions.f90:777-918 + structure(), or the weighted form of
// src/BoundaryConditions3.f90:777-903) and the fault SAT computed by the
// interface kernel (src/RHS_Interior.f90:1757-1772) of each face point, tot,
// folded into the rates before the stencil kernel runs, DF <- DF - tot/A, or
// DF <- -tot on a stage with A = 0, so that the stencil's A*DF + du (or
// DF + du on face points when A = 0) carries it.  On a PML side the same
// boundary forcing enters the rates of the slab's auxiliary fields
// (src/RHS_Interior.f90:1560-1700): it is folded into DQ in the same way,
// for the PML pre-kernel to pick up.  One thread per face point, a point on
// several faces taken by its lowest side.
template <typename T, bool PML>
__device__ __forceinline__ void face_pre_point(const VolumeArgs<T>& a, long long t) {
  const int nq = a.nq, nr = a.nr, ns = a.ns;
  const long long nfs[6] = {(long long)nr * ns, (long long)nr * ns, (long long)nq * ns, (long long)nq * ns,
                            (long long)nq * nr, (long long)nq * nr};
  int side = 0;
  while (side < 6 && t >= nfs[side]) {
    t -= nfs[side];
    ++side;
  }
  if (side >= 6) return;
  const int axis = side >> 1;
  const int w = axis == 0 ? nr : nq;
  const int c2 = (int)((unsigned)t / (unsigned)w), c1 = (int)((unsigned)t - (unsigned)c2 * (unsigned)w);
  int i, j, k;
  if (axis == 0) { i = (side & 1) ? nq - 1 : 0; j = c1; k = c2; }
  else if (axis == 1) { i = c1; j = (side & 1) ? nr - 1 : 0; k = c2; }
  else { i = c1; j = c2; k = (side & 1) ? ns - 1 : 0; }
  for (int s2 = 0; s2 < side; ++s2) {
    const int ax2 = s2 >> 1;
    const int ii = ax2 == 0 ? i : (ax2 == 1 ? j : k), n2 = ax2 == 0 ? nq : (ax2 == 1 ? nr : ns);
    if (ii == ((s2 & 1) ? n2 - 1 : 0)) return;
  }
  const long long np = a.np;
  const long long p = i + (long long)a.pq * (j + (long long)nr * k);
  T u[9], tot[9], df[9];
  // the rates are read together with the fields (not after the penalty is
  // formed), so the two loads' latencies overlap; a stage with A = 0
  // overwrites them without reading
  const bool keep = a.A != T(0);
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    u[c] = a.Fin[c * np + p];
    df[c] = keep ? a.DF[c * np + p] : T(0);
  }
  mms_deviation(a, p, u);
  face_penalty(a, i, j, k, u, tot, [&](int s2, const T (&ubc)[9]) {
    if (!PML || !a.pml[s2]) return;
    const long long sp = slab_point(a, s2, i, j, k), snp = a.slab_np[s2];
    const T th = a.tau_h[s2 >> 1];
    T* DQ = a.DQ[s2];
#pragma unroll
    for (int c = 0; c < 9; ++c) DQ[c * snp + sp] = keep ? DQ[c * snp + sp] - th * ubc[c] * a.Ainv : -th * ubc[c];
  });
  // a face point without a penalised side still defines DF when A = 0
#pragma unroll
  for (int c = 0; c < 9; ++c) a.DF[c * np + p] = df[c] - tot[c] * a.Ainv;
}

// One launch covers one block or both of a scenario: threads [0, n0) take
// block 0's face points, the rest block 1's (one launch of about twice the
// threads hides the latency of these sub-wave launches better than two).
// PML: some side has a slab.
template <typename T, bool PML>
__global__ void __launch_bounds__(256) face_pre_kernel(const __grid_constant__ BlockPair<T> P) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t < P.n0) face_pre_point<T, PML>(P.a[0], t);
  else face_pre_point<T, PML>(P.a[1], t - P.n0);
}

// ---------------------------------------------------------------------------
// Moment-tensor point source (set_moment_tensor / set_moment_tensor_smooth,
// src/moment_tensor.f90:1014-1078, 1400-1475): DF(4:9) -= (A(t) M) * delta
// on the source's box of points, with the matching update of F_out.
struct SourceArgs {
  int lo[3], dim[3];
  const double* delta;
  double am[6];
};

template <typename T, bool KAHAN>
__global__ void __launch_bounds__(256) source_kernel(const __grid_constant__ VolumeArgs<T> a,
                                                     const __grid_constant__ SourceArgs s) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long n = (long long)s.dim[0] * s.dim[1] * s.dim[2];
  if (e >= n) return;
  const int i = s.lo[0] + (int)(e % s.dim[0]);
  const int j = s.lo[1] + (int)((e / s.dim[0]) % s.dim[1]);
  const int k = s.lo[2] + (int)(e / ((long long)s.dim[0] * s.dim[1]));
  const long long p = i + (long long)a.pq * (j + (long long)a.nr * k);
  const double d = s.delta[e];
  T corr[9];
#pragma unroll
  for (int c = 0; c < 3; ++c) corr[c] = T(0);
#pragma unroll
  for (int c = 0; c < 6; ++c) corr[3 + c] = (T)(-(s.am[c] * d));
  add_correction<T, KAHAN>(a, p, corr);
}

// ---------------------------------------------------------------------------
// Plastic return map after the last stage (update_fields_plastic,
// src/plastic.f90:11-151: plastic_flow2 :153-217 for plastic_model 'scec',
// plastic_flow :220-290 otherwise), on points outside the PML slabs,
// applied to the updated stresses.
// The grid covers the box outside the slabs, [lo, hi) per axis; the
// uniform constants come in the field type (pc: c cos(atan nu), sin(atan nu),
// exp(-dt/Tv); s0: the uniform initial stress), so no thread converts from
// FP64.
template <typename T>
struct PlasticBox {
  int lo[3], hi[3];
  T pc[3];
  T s0[6];
};

template <typename T, bool CURV, bool KAHAN>
__global__ void __launch_bounds__(256) plastic_kernel(const __grid_constant__ VolumeArgs<T> a,
                                                      const __grid_constant__ PlasticBox<T> box) {
  const int i = box.lo[0] + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = box.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = box.lo[2] + blockIdx.z;
  if (i >= box.hi[0] || j >= box.hi[1]) return;
  const long long np = a.np;
  const long long p = i + (long long)a.pq * (j + (long long)a.nr * k);
  T s0[6];
  if (!initial_stress_y<T>(a.preset, a.ycoord[p], s0))
    for (int c = 0; c < 6; ++c) s0[c] = box.s0[c];
  T sa[6];
  for (int c = 0; c < 6; ++c) sa[c] = a.Fout[(3 + c) * np + p] + s0[c];
  const T sigma = (sa[0] + sa[1] + sa[2]) / T(3);
  const T J2 = ((sa[0] - sa[1]) * (sa[0] - sa[1]) + (sa[1] - sa[2]) * (sa[1] - sa[2]) +
                (sa[2] - sa[0]) * (sa[2] - sa[0])) / T(6) +
               sa[3] * sa[3] + sa[4] * sa[4] + sa[5] * sa[5];
  const T tau = sqrt(J2);
  if (a.pl_flow) {
    // plastic_flow (src/plastic.f90:220-290): yield function Y = tau + mu*sigma;
    // above it the closed-form solution of eta*lambda = Y(s) for the plastic
    // strain rate, with shear modulus G and bulk modulus K of the point
    const T mu = (T)a.pl_mu, beta = (T)a.pl_beta, eta = (T)a.pl_eta, dt = (T)a.dt;
    const T Y = tau + mu * sigma;
    if (Y <= T(0)) {
      a.pl_lambda[p] = T(0);
      return;
    }
    const T* coef = a.coef;
    const T G = CURV ? coef[11 * np + p] : coef[1 * np + p];
    const T K = (CURV ? coef[10 * np + p] : coef[0 * np + p]) + T(2.0 / 3.0) * G;
    T sd[6];
    for (int c = 0; c < 6; ++c) sd[c] = sa[c] - sigma * (c < 3 ? T(1) : T(0));
    const T lambda = (tau + mu * sigma) / (eta + dt * (G + mu * beta * K));
    a.pl_lambda[p] = lambda;
    a.pl_gammap[p] = a.pl_gammap[p] + dt * lambda;
    const T tau1 = tau - dt * lambda * G;
    const T sigma1 = sigma - dt * lambda * beta * K;
    for (int c = 0; c < 6; ++c) {
      const T sdc = sd[c] * tau1 / (tau1 + dt * lambda * G);
      a.Fout[(3 + c) * np + p] = (sigma1 * (c < 3 ? T(1) : T(0)) + sdc) - s0[c];
      if (KAHAN) a.C[(3 + c) * np + p] = 0;  // bfloat16 zero
    }
    return;
  }
  // c cos(atan nu), sin(atan nu) and exp(-dt/Tv) are uniform: set on the host
  const T Ys = fmax(T(0), box.pc[0] - sigma * box.pc[1]);
  if (!(tau - Ys > T(0))) return;
  const T e = box.pc[2];
  const T rr = e + (T(1) - e) * Ys / tau;
  for (int c = 0; c < 6; ++c) {
    const T dlt = c < 3 ? T(1) : T(0);
    const T sd = sa[c] - sigma * dlt;
    a.Fout[(3 + c) * np + p] = (sigma * dlt + rr * sd) - s0[c];
    if (KAHAN) a.C[(3 + c) * np + p] = 0;  // bfloat16 zero
  }
}

}  // namespace

template <typename T, bool CURV, bool KAHAN, int TQ, int TR, int MINB>
void launch_tiled(const VolumeArgs<T>& a, cudaStream_t s) {
  const size_t smem = sizeof(T) * Tile<T, TQ, TR>::words;
  auto kern = stencil_kernel_tiled<T, CURV, KAHAN, TQ, TR, MINB>;
  static bool attr_done = false;
  if (!attr_done) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr_done = true;
  }
  const int schunk = a.schunk > 0 ? a.schunk : 16;
  dim3 blk(TQ, TR, 1), grd((a.nq + TQ - 1) / TQ, (a.nr + TR - 1) / TR, (a.ns + schunk - 1) / schunk);
  kern<<<grd, blk, smem, s>>>(a, schunk);
}

// Stencil-kernel variants (the tuning table): 1 per-point, 2 tiled 32x8 at
// 1 CTA/SM, 3 tiled 32x8 at 3 CTAs/SM in FP32, 4 tiled 64x8 at 1 CTA/SM,
// 5 TMA-pipelined (FP32), 6 accepted as 5; 0 picks the TMA kernel in FP32
// and in FP64 the kernel of wql_stencil_fp64.cu (7 here; a block that no split
// fits, 22 x 17 points in q and r alone up to 420, takes the tiled kernel).
//
// Axes whose closure rows a tile would not hold (tiles_ok, tiles_ok_up) run per
// point.

// Rows of the TMA tiles that the block's tensor maps are shaped for.
template <typename T>
int tma_tile_rows(const VolumeArgs<T>& a) {
  return tma_rows(a.tma ? static_cast<const StencilMaps*>(a.tma)->tq : kTmaTQ);
}

template <typename T>
int effective_variant(const VolumeArgs<T>& a) {
  constexpr bool f32 = sizeof(T) == 4;
  int v = a.kernel != 0 ? a.kernel : (f32 ? 5 : (a.plan64 && a.plan64->ok && !a.fd ? 7 : 2));
  if ((v == 5 || v == 6) && !(f32 && a.C != nullptr)) v = 2;
  if (a.fd) {
    // the order-6 upwind pair: the TMA kernel (compensated FP32) or per
    // point; order 5 per point
    if (a.fd != 1 || !(v == 5 || v == 6) || a.C == nullptr || !tiles_ok_up(a.nr, tma_tile_rows(a))) v = 1;
    return v;
  }
  if ((v == 5 || v == 6) && !tiles_ok(a.nr, tma_tile_rows(a))) v = 1;
  if ((v == 2 || v == 3) && !(tiles_ok(a.nq, 32) && tiles_ok(a.nr, 8))) v = 1;
  if (v == 4 && !(tiles_ok(a.nq, 64) && tiles_ok(a.nr, 8))) v = 1;
  return v;
}

// Whether the block's stencil runs as the TMA kernel.
template <typename T>
bool stencil_is_tma(const VolumeArgs<T>& a) {
  const int v = effective_variant(a);
  return v == 5 || v == 6;
}

template <typename T, bool CURV, bool KAHAN>
void launch_pointwise(const VolumeArgs<T>& a0, const VolumeArgs<T>* a1, cudaStream_t s) {
  BlockPair<T> P;
  P.a[0] = a0;
  P.a[1] = a1 ? *a1 : a0;
  P.n0 = a0.ns;
  // 16 x 8 points: few idle lanes on short rows, and the q closure columns stay
  // in fewer warps (upwind-DRP 6 on 2 x 76x101x91: 1.13 ms a step; 16 x 16 1.14,
  // 32 x 8 1.19, 8 x 16 1.34)
  dim3 blk(16, 8, 1), grd((std::max(a0.nq, P.a[1].nq) + 15) / 16, (a0.nr + 7) / 8, a0.ns + (a1 ? a1->ns : 0));
  switch (a0.fd) {
    case 0: stencil_kernel_pointwise<T, CURV, KAHAN, 0><<<grd, blk, 0, s>>>(P); return;
    case 1: stencil_kernel_pointwise<T, CURV, KAHAN, 1><<<grd, blk, 0, s>>>(P); return;
    case 2: stencil_kernel_pointwise<T, CURV, KAHAN, 2><<<grd, blk, 0, s>>>(P); return;
    default: break;
  }
  switch (ug_window(a0.ug)) {
    case 3: stencil_kernel_pointwise<T, CURV, KAHAN, 3><<<grd, blk, 0, s>>>(P); return;
    case 4: stencil_kernel_pointwise<T, CURV, KAHAN, 4><<<grd, blk, 0, s>>>(P); return;
    default: stencil_kernel_pointwise<T, CURV, KAHAN, 5><<<grd, blk, 0, s>>>(P); return;
  }
}

template <typename T, bool CURV, bool KAHAN>
void launch_stencil(const VolumeArgs<T>& a, cudaStream_t s) {
  constexpr bool f32 = sizeof(T) == 4;
  const int v = effective_variant(a);
  switch (v) {
    case 1: launch_pointwise<T, CURV, KAHAN>(a, nullptr, s); return;
    case 3: launch_tiled<T, CURV, KAHAN, 32, 8, f32 ? 3 : 1>(a, s); return;
    case 4: launch_tiled<T, CURV, KAHAN, 64, 8, 1>(a, s); return;
    case 5:
    case 6:
      if constexpr (f32 && KAHAN) {
        launch_stencil_tma(a, CURV, s);
        return;
      }
      [[fallthrough]];
    case 7:
      if constexpr (!f32) {
        launch_stencil_fp64(a, nullptr, CURV, s);
        return;
      }
      [[fallthrough]];
    default: launch_tiled<T, CURV, KAHAN, 32, 8, 1>(a, s); return;
  }
}

template <typename T, bool CURV, bool KAHAN>
int launch_corr(const VolumeArgs<T>& a, cudaStream_t s) {
  int n = 0;
  dim3 blk(32, 8, 1), grd((a.nq + 31) / 32, (a.nr + 7) / 8, a.ns);
  if (a.anel && a.G == nullptr) {
    if (a.fd == 1) anelastic_kernel<T, CURV, KAHAN, 1><<<grd, blk, 0, s>>>(a);
    else if (a.fd == 2) anelastic_kernel<T, CURV, KAHAN, 2><<<grd, blk, 0, s>>>(a);
    else if (a.fd == 3) anelastic_kernel<T, CURV, KAHAN, 5><<<grd, blk, 0, s>>>(a);
    else anelastic_kernel<T, CURV, KAHAN, 0><<<grd, blk, 0, s>>>(a);
    ++n;
  } else if (a.anel) {
    anelastic_comp_kernel<T, CURV, KAHAN><<<(unsigned)((a.np + 63) / 64), 384, 0, s>>>(a);
    ++n;
  }
  if (a.mp) {
    mms_kernel<T, KAHAN><<<grd, blk, 0, s>>>(a);
    ++n;
  }
  if (a.plastic) {
    PlasticBox<T> box;
    const int nn[3] = {a.nq, a.nr, a.ns};
    for (int ax = 0; ax < 3; ++ax) {
      box.lo[ax] = a.pml[2 * ax] ? a.npml : 0;
      box.hi[ax] = a.pml[2 * ax + 1] ? nn[ax] - a.npml : nn[ax];
    }
    box.pc[0] = (T)a.pl_ccos;
    box.pc[1] = (T)a.pl_sin;
    box.pc[2] = (T)a.pl_decay;
    for (int c = 0; c < 6; ++c) box.s0[c] = (T)a.s0u[c];
    const int bq = box.hi[0] - box.lo[0], br = box.hi[1] - box.lo[1], bs = box.hi[2] - box.lo[2];
    if (bq > 0 && br > 0 && bs > 0) {
      dim3 pgrd((bq + 31) / 32, (br + 7) / 8, bs);
      plastic_kernel<T, CURV, KAHAN><<<pgrd, blk, 0, s>>>(a, box);
    }
    ++n;
  }
  return n;
}

template <typename T>
void launch_volume(const VolumeArgs<T>& a, bool curv, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const bool kahan = a.C != nullptr;
  if (curv) kahan ? launch_stencil<T, true, true>(a, s) : launch_stencil<T, true, false>(a, s);
  else kahan ? launch_stencil<T, false, true>(a, s) : launch_stencil<T, false, false>(a, s);
}

template <typename T>
int launch_pre(const VolumeArgs<T>& a0, const VolumeArgs<T>* a1, bool curv, void* stream) {
  BlockPair<T> P;
  P.a[0] = a0;
  P.a[1] = a1 ? *a1 : a0;
  auto nface = [](const VolumeArgs<T>& a) {
    return 2LL * ((long long)a.nr * a.ns + (long long)a.nq * a.ns + (long long)a.nq * a.nr);
  };
  P.n0 = nface(a0);
  const long long n = P.n0 + (a1 ? nface(*a1) : 0);
  const unsigned g = (unsigned)((n + 255) / 256);
  if (a0.npml > 0 || (a1 && a1->npml > 0)) face_pre_kernel<T, true><<<g, 256, 0, (cudaStream_t)stream>>>(P);
  else face_pre_kernel<T, false><<<g, 256, 0, (cudaStream_t)stream>>>(P);
  return 1 + launch_pml_pre(a0, a1, curv, (cudaStream_t)stream);
}

template <typename T>
int launch_volume2(const VolumeArgs<T>& a0, const VolumeArgs<T>& a1, bool curv, void* stream) {
  const int v = effective_variant(a0);
  if (v != effective_variant(a1) || !(v == 1 || v == 5 || v == 6 || v == 7)) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const bool kahan = a0.C != nullptr;
  if (v == 1) {
    if (a0.nr != a1.nr || a0.ns + a1.ns > 65535) return 0;  // one grid over both blocks' planes
    if (curv) kahan ? launch_pointwise<T, true, true>(a0, &a1, s) : launch_pointwise<T, true, false>(a0, &a1, s);
    else kahan ? launch_pointwise<T, false, true>(a0, &a1, s) : launch_pointwise<T, false, false>(a0, &a1, s);
    return 1;
  }
  if constexpr (sizeof(T) == 4) launch_stencil_tma2(a0, a1, curv, stream);
  else launch_stencil_fp64(a0, &a1, curv, stream);
  return 1;
}

template <typename T>
int launch_corrections(const VolumeArgs<T>& a0, bool curv, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  // the velocity gradient of an anelastic block comes from the stencil only
  // when that was the TMA kernel (the only one that writes it)
  VolumeArgs<T> a = a0;
  if (!stencil_is_tma(a)) a.G = nullptr;
  const bool kahan = a.C != nullptr;
  if (curv) return kahan ? launch_corr<T, true, true>(a, s) : launch_corr<T, true, false>(a, s);
  return kahan ? launch_corr<T, false, true>(a, s) : launch_corr<T, false, false>(a, s);
}

template <typename T>
void launch_source(const VolumeArgs<T>& a, const int lo[3], const int dim[3], const double* delta,
                   const double am[6], void* stream) {
  SourceArgs s;
  for (int c = 0; c < 3; ++c) {
    s.lo[c] = lo[c];
    s.dim[c] = dim[c];
  }
  for (int c = 0; c < 6; ++c) s.am[c] = am[c];
  s.delta = delta;
  const long long n = (long long)dim[0] * dim[1] * dim[2];
  if (n <= 0) return;
  const unsigned g = (unsigned)((n + 255) / 256);
  if (a.C) source_kernel<T, true><<<g, 256, 0, (cudaStream_t)stream>>>(a, s);
  else source_kernel<T, false><<<g, 256, 0, (cudaStream_t)stream>>>(a, s);
}

template void launch_source<double>(const VolumeArgs<double>&, const int*, const int*, const double*,
                                    const double*, void*);
template void launch_source<float>(const VolumeArgs<float>&, const int*, const int*, const double*,
                                   const double*, void*);
template void launch_volume<double>(const VolumeArgs<double>&, bool, void*);
template void launch_volume<float>(const VolumeArgs<float>&, bool, void*);
template int launch_corrections<double>(const VolumeArgs<double>&, bool, void*);
template int launch_pre<double>(const VolumeArgs<double>&, const VolumeArgs<double>*, bool, void*);
template int launch_pre<float>(const VolumeArgs<float>&, const VolumeArgs<float>*, bool, void*);
template int launch_volume2<double>(const VolumeArgs<double>&, const VolumeArgs<double>&, bool, void*);
template int launch_volume2<float>(const VolumeArgs<float>&, const VolumeArgs<float>&, bool, void*);
template int launch_corrections<float>(const VolumeArgs<float>&, bool, void*);
template bool stencil_is_tma<float>(const VolumeArgs<float>&);
template bool stencil_is_tma<double>(const VolumeArgs<double>&);

}  // namespace wql
